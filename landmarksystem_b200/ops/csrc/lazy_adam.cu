// Lazy (deferred) Adam for feature planes: exact Adam semantics at a fraction of the memory traffic.
//
// A training step touches only the texels its samples fall on (about a quarter of a 4096^2 plane for
// 10^6 samples), yet a dense Adam pass reads and writes every parameter and both moments each step
// (34 bytes per parameter; 36 GB per step for a 10^9-parameter grid, which dominated the step).  With
// zero gradient the Adam recurrence of an element needs nothing but its own state,
//     m <- b1 m,  v <- b2 v,  p <- p - lr_k / (1 - b1^k) * m / (sqrt(v / (1 - b2^k)) + eps),
// so an untouched texel can be left alone and caught up later by replaying the skipped steps in
// registers.  Per step:
//   mark     every texel the step's samples will read gets need = 1                         (vm_mark)
//   prepare  needed texels that are behind get their bf16 shadow value brought to "after step t-1"
//            (reads p, m, v; writes only the 2-byte shadow)
//   step     after backward, needed texels replay their skipped steps, apply step t with the real
//            gradient, store p / m / v / shadow once, clear the gradient and record last_step = t
//   flush    brings every texel up to date (before checkpoints, evaluation, resizing).
// The learning-rate schedule is the trainers' geometric decay: lr_k = lr_t * decay^(k - t).
#include "common.cuh"
#include <cmath>

namespace lmb {

struct LazySched {
  float lr_ref;    // learning rate of step t_ref
  int t_ref;
  float decay;     // lr_{k+1} = lr_k * decay
  float beta1, beta2, eps;
  float l2_decay, l2_beta1, l2_beta2;   // log2 of the three bases (host, double precision)
  int t;           // step being prepared / applied, or (flush) the last completed step (1-based)
  const float* dyn;  // optional device-resident {lr of the step being applied, its number}: overrides lr_ref, t_ref, t
};

__device__ __forceinline__ void resolve_dyn(LazySched& s) {
  if (s.dyn != nullptr) {
    s.lr_ref = s.dyn[0];
    s.t_ref = s.t = (int)s.dyn[1];
  }
}

struct Replay {
  float lr, b1p, b2p;   // lr_k, beta1^k, beta2^k of the NEXT step to replay
};

__device__ __forceinline__ Replay replay_start(const LazySched& s, int k) {
  Replay r;
  r.lr = s.lr_ref * exp2f(s.l2_decay * (float)(k - s.t_ref));
  r.b1p = exp2f(s.l2_beta1 * (float)k);
  r.b2p = exp2f(s.l2_beta2 * (float)k);
  return r;
}

// advance one zero-gradient step for 4 elements
__device__ __forceinline__ void zero_grad_step(float4& p, float4& m, float4& v, const LazySched& s, Replay& r) {
  const float step = r.lr / (1.f - r.b1p);
  const float inv_sqrt_b2 = rsqrtf(1.f - r.b2p);
  float* P = &p.x; float* M = &m.x; float* V = &v.x;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    M[k] *= s.beta1;
    V[k] *= s.beta2;
    P[k] -= step * M[k] / (sqrtf(V[k]) * inv_sqrt_b2 + s.eps);
  }
  r.lr *= s.decay; r.b1p *= s.beta1; r.b2p *= s.beta2;
}

// The same where `on`, nothing elsewhere, without a branch and without a second copy of the state: factors of one leave the
// moments as they are.
__device__ __forceinline__ void zero_grad_step_if(bool on, float4& p, float4& m, float4& v, const LazySched& s, Replay& r) {
  const float step = r.lr / (1.f - r.b1p);
  const float inv_sqrt_b2 = rsqrtf(1.f - r.b2p);
  const float b1 = on ? s.beta1 : 1.f, b2 = on ? s.beta2 : 1.f;
  float* P = &p.x; float* M = &m.x; float* V = &v.x;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    M[k] *= b1;
    V[k] *= b2;
    const float next = P[k] - step * M[k] / (sqrtf(V[k]) * inv_sqrt_b2 + s.eps);
    P[k] = on ? next : P[k];
  }
  r.lr *= on ? s.decay : 1.f; r.b1p *= b1; r.b2p *= b2;
}

__device__ __forceinline__ uint2 to_bf16x4(const float4& p) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y), hi = __floats2bfloat162_rn(p.z, p.w);
  uint2 u;
  u.x = *reinterpret_cast<unsigned*>(&lo); u.y = *reinterpret_cast<unsigned*>(&hi);
  return u;
}

// need: 0 idle, 1 marked, 2 prepared.
constexpr int kMaxReplay = 192;   // beta1^192 < 2e-9: later zero-gradient steps cannot change an fp32 parameter

// number of zero-gradient steps to run explicitly / to fold into a moment decay afterwards
__device__ __forceinline__ void replay_plan(int last, int upto, int& n_explicit, int& n_rest) {
  const int n = (last == 0 || upto <= last) ? 0 : upto - last;   // never stepped: both moments are zero and stay zero
  n_explicit = n < kMaxReplay ? n : kMaxReplay;
  n_rest = n - n_explicit;
}
__device__ __forceinline__ void decay_moments(float4& mm, float4& vv, const LazySched& s, int n_rest) {
  if (n_rest > 0) {                               // the remaining steps only decay the moments
    const float d1 = exp2f(s.l2_beta1 * (float)n_rest), d2 = exp2f(s.l2_beta2 * (float)n_rest);
    mm.x *= d1; mm.y *= d1; mm.z *= d1; mm.w *= d1;
    vv.x *= d2; vv.y *= d2; vv.z *= d2; vv.w *= d2;
  }
}

// Bound by memory: p, m, v (and g) of the flagged texels in, p, m, v, g and the shadow out, one flag byte per texel; warps wait for
// the scattered loads at 51 % of the DRAM rate (4096^2 texels of 16 channels, 28 warps an SM).  A warp
// walks the flags 32 kPer texels at a time, lists the flagged ones in texel order in shared memory and spreads their (texel,
// 4-channel group) items over its lanes, so that a texel's channels move as one contiguous run and addresses only ever
// increase.  A step flags 5 - 25 % of a large plane: of 32 texels too few to fill a warp's requests (16 channels: 13 of 32
// lanes), of 128 enough.  The next flags are fetched while the current texels are processed.  4096^2 texels, 16 and 48 channels
// together, 8192 rays: step 920 -> 731 us, prepare 582 -> 431 us.
constexpr int kLazyWarps = 8;

template <int kPer>
__device__ __forceinline__ uint32_t load_flags(const unsigned char* __restrict__ need, long long texel, long long n_texels) {
  if (kPer == 4 && texel + 4 <= n_texels) return *reinterpret_cast<const uint32_t*>(need + texel);
  uint32_t f = 0;
  for (int k = 0; k < kPer; ++k)
    if (texel + k < n_texels) f |= (uint32_t)need[texel + k] << (8 * k);
  return f;
}

template <bool kPrepare, int kPer>
__global__ void __launch_bounds__(32 * kLazyWarps)
lazy_scan_kernel(unsigned char* __restrict__ need, int* __restrict__ last_step, float4* __restrict__ p, float4* __restrict__ g,
                 float4* __restrict__ m, float4* __restrict__ v, uint2* __restrict__ shadow, int c4, long long n_texels,
                 LazySched s, float grad_scale) {
  constexpr int kChunk = 32 * kPer;
  __shared__ unsigned char s_list[kLazyWarps][kChunk];
  resolve_dyn(s);
  const int lane = threadIdx.x & 31;
  unsigned char* list = s_list[threadIdx.x >> 5];
  const long long stride = (long long)gridDim.x * kLazyWarps * kChunk;
  const int which_step = 32 / c4, grp_step = 32 - which_step * c4, which0 = lane / c4, grp0 = lane - which0 * c4;
  long long base = ((long long)blockIdx.x * kLazyWarps + (threadIdx.x >> 5)) * kChunk;
  uint32_t ahead = base < n_texels ? load_flags<kPer>(need, base + kPer * lane, n_texels) : 0u;
  for (; base < n_texels; base += stride) {
    const uint32_t flags = ahead;
    const long long texel = base + kPer * lane;
    ahead = base + stride < n_texels ? load_flags<kPer>(need, texel + stride, n_texels) : 0u;
    uint32_t mine = 0, work = 0;                                  // one bit per texel of this lane
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t f = flags >> (8 * k) & 0xFF;
      if (kPrepare ? f == 1 : f != 0) mine |= 1u << k;
    }
    if (kPrepare) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int last = mine >> k & 1 ? last_step[texel + k] : 0;
        if (last > 0 && last < s.t - 1) work |= 1u << k;
      }
    } else {
      work = mine;
    }
    int at = __popc(work);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, at, d);
      if (lane >= d) at += below;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31) * c4;
    at -= __popc(work);
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (work >> k & 1) list[at++] = (unsigned char)(kPer * lane + k);
    __syncwarp();
    // Every lane runs every statement below (loads, stores and arithmetic are predicated on `on`): the
    // replay loop has ONE trip count per warp, so lanes never split and each memory instruction is issued
    // once per warp with all its addresses together.
    int which = which0, grp = grp0;
    for (int w0 = 0; w0 < total; w0 += 32) {
      const bool on = w0 + lane < total;
      const long long t = base + (on ? list[which] : 0);
      const long long e = t * c4 + grp;
      const int last_t = on ? last_step[t] : 0;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 pp = on ? p[e] : zero, mm = on ? m[e] : zero, vv = on ? v[e] : zero;
      float4 gg = zero;
      if (!kPrepare && on) gg = g[e];
      which += which_step; grp += grp_step;
      if (grp >= c4) { grp -= c4; ++which; }
      int n_explicit, n_rest;
      replay_plan(last_t, s.t - 1, n_explicit, n_rest);
      const int n_warp = __reduce_max_sync(0xffffffffu, n_explicit);
      Replay r = replay_start(s, last_t + 1);
      for (int k = 0; k < n_warp; ++k) zero_grad_step_if(k < n_explicit, pp, mm, vv, s, r);
      decay_moments(mm, vv, s, n_rest);
      if (kPrepare) {
        if (on) shadow[e] = to_bf16x4(pp);
      } else {
        Replay rt = replay_start(s, s.t);
        const float step = rt.lr / (1.f - rt.b1p);
        const float inv_sqrt_b2 = rsqrtf(1.f - rt.b2p);
        const float* G = &gg.x; float* P = &pp.x; float* M = &mm.x; float* V = &vv.x;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float gr = G[k] * grad_scale;
          M[k] = s.beta1 * M[k] + (1.f - s.beta1) * gr;
          V[k] = s.beta2 * V[k] + (1.f - s.beta2) * gr * gr;
          P[k] -= step * M[k] / (sqrtf(V[k]) * inv_sqrt_b2 + s.eps);
        }
        if (on) {
          g[e] = zero;
          p[e] = pp; m[e] = mm; v[e] = vv;
          if (shadow) shadow[e] = to_bf16x4(pp);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (mine >> k & 1) {
        need[texel + k] = kPrepare ? 2 : 0;
        if (!kPrepare) last_step[texel + k] = s.t;
      }
  }
}

// flush: every texel of the plane that is behind step s.t replays up to it (no gradient); one thread
// per (texel, group), last_step is advanced by a second launch
__global__ void __launch_bounds__(256)
lazy_flush_kernel(const int* __restrict__ last_step, float4* __restrict__ p, float4* __restrict__ m, float4* __restrict__ v,
                  uint2* __restrict__ shadow, int c4, long long n_texels, LazySched s) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long texel = e / c4;
  if (texel >= n_texels) return;
  const int last = last_step[texel];
  if (last >= s.t || last == 0) return;
  float4 pp = p[e], mm = m[e], vv = v[e];
  int n_explicit, n_rest;
  replay_plan(last, s.t, n_explicit, n_rest);
  Replay r = replay_start(s, last + 1);
  for (int k = 0; k < n_explicit; ++k) zero_grad_step(pp, mm, vv, s, r);
  decay_moments(mm, vv, s, n_rest);
  p[e] = pp; m[e] = mm; v[e] = vv;
  if (shadow) shadow[e] = to_bf16x4(pp);
}
__global__ void __launch_bounds__(256) lazy_flush_commit_kernel(int* __restrict__ last_step, long long n_texels, int t) {
  const long long texel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (texel < n_texels && last_step[texel] < t) last_step[texel] = t;
}

// Flag the 4 corner texels of every sample on one plane level (same tap rule as the lookup kernel).
__global__ void __launch_bounds__(256)
vm_mark_kernel(const float4* __restrict__ coords, const int* __restrict__ count_ptr, long long max_n, int B, int H, int W,
               unsigned char* __restrict__ need) {
  const long long n_valid = resolve_count(count_ptr, max_n);
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_valid) return;
  const float4 q = __ldg(coords + n);
  const int b = (int)q.w;
  if (b < 0 || b >= B) return;
  const float fx = (q.x + 1.f) * 0.5f * (float)(W - 1), fy = (q.y + 1.f) * 0.5f * (float)(H - 1);
  const int x0 = (int)floorf(fx), y0 = (int)floorf(fy);
#pragma unroll
  for (int corner = 0; corner < 4; ++corner) {
    const int x = min(max(x0 + (corner & 1), 0), W - 1), y = min(max(y0 + (corner >> 1), 0), H - 1);
    unsigned char* f = need + ((long long)b * H + y) * W + x;
    if (*f == 0) *f = 1;
  }
}

}  // namespace lmb

using namespace lmb;

static LazySched make_sched(float lr_ref, int t_ref, float decay, float beta1, float beta2, float eps, int t,
                            const float* dyn = nullptr) {
  LazySched s;
  s.dyn = dyn;
  s.lr_ref = lr_ref; s.t_ref = t_ref; s.decay = decay; s.beta1 = beta1; s.beta2 = beta2; s.eps = eps; s.t = t;
  s.l2_decay = (float)log2((double)decay); s.l2_beta1 = (float)log2((double)beta1); s.l2_beta2 = (float)log2((double)beta2);
  return s;
}

// Texels per lane: chunks of 128 texels fill a warp's requests, but there must be one for every warp that the GPU holds
// (148 x 32); a smaller plane is cut finer, and most of it is flagged by a step anyway.  Prepare + step of a 16- and a
// 48-channel plane, 8192 rays, 128 against 32 texels: 512^2 texels 124 against 96 us, 700^2 146 against 141, 1000^2 212 against
// 227, 1300^2 267 against 300.
constexpr long long kLargePlane = 148LL * 32 * 128;

template <bool kPrepare>
static int launch_scan(unsigned char* need, int* last_step, float* p, float* g, float* m, float* v, void* shadow, int C,
                       long long n_texels, const LazySched& s, float grad_scale, cudaStream_t stream) {
  const bool large = n_texels >= kLargePlane && (uintptr_t)need % 4 == 0;      // flags are then read as 4-byte words
  const auto kernel = large ? lazy_scan_kernel<kPrepare, 4> : lazy_scan_kernel<kPrepare, 1>;
  const long long per_block = kLazyWarps * 32 * (large ? 4 : 1), blocks = (n_texels + per_block - 1) / per_block;
  const long long cap = 148 * (large ? 16 : 32);
  kernel<<<(int)(blocks < cap ? blocks : cap), 32 * kLazyWarps, 0, stream>>>(need, last_step, (float4*)p, (float4*)g, (float4*)m,
                                                                            (float4*)v, (uint2*)shadow, C / 4, n_texels, s, grad_scale);
  LMB_LAUNCH_CHECK();
  return 0;
}

// need: uint8 [B*H*W]
LMB_API int lmb_vm_mark(const float* coords, const int* count_ptr, long long max_n, int B, int H, int W, unsigned char* need,
                        cudaStream_t stream) {
  if (max_n <= 0) return 0;
  vm_mark_kernel<<<ceil_div(max_n, 256), 256, 0, stream>>>((const float4*)coords, count_ptr, max_n, B, H, W, need);
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API int lmb_lazy_adam_prepare(unsigned char* need, int* last_step, const float* p, const float* m, const float* v,
                                  void* shadow, int C, long long n_texels, float lr_ref, int t_ref, float decay, float beta1,
                                  float beta2, float eps, int t, const float* dyn, cudaStream_t stream) {
  if (C % 4) return (int)cudaErrorInvalidValue;
  if (n_texels <= 0) return 0;
  return launch_scan<true>(need, last_step, const_cast<float*>(p), nullptr, const_cast<float*>(m), const_cast<float*>(v), shadow, C,
                           n_texels, make_sched(lr_ref, t_ref, decay, beta1, beta2, eps, t, dyn), 1.f, stream);
}

LMB_API int lmb_lazy_adam_step(unsigned char* need, int* last_step, float* p, float* g, float* m, float* v, void* shadow,
                               int C, long long n_texels, float lr_ref, int t_ref, float decay, float beta1, float beta2,
                               float eps, int t, float grad_scale, const float* dyn, cudaStream_t stream) {
  if (C % 4) return (int)cudaErrorInvalidValue;
  if (n_texels <= 0) return 0;
  return launch_scan<false>(need, last_step, p, g, m, v, shadow, C, n_texels,
                            make_sched(lr_ref, t_ref, decay, beta1, beta2, eps, t, dyn), grad_scale, stream);
}

// Bring every texel up to step t (zero-gradient replay); call between steps (no flags set).
LMB_API int lmb_lazy_adam_flush(int* last_step, float* p, float* m, float* v, void* shadow, int C, long long n_texels,
                                float lr_ref, int t_ref, float decay, float beta1, float beta2, float eps, int t,
                                cudaStream_t stream) {
  if (C % 4) return (int)cudaErrorInvalidValue;
  if (n_texels <= 0) return 0;
  const int c4 = C / 4;
  lazy_flush_kernel<<<ceil_div(n_texels * c4, 256), 256, 0, stream>>>(last_step, (float4*)p, (float4*)m, (float4*)v,
                                                                     (uint2*)shadow, c4, n_texels,
                                                                     make_sched(lr_ref, t_ref, decay, beta1, beta2, eps, t));
  LMB_LAUNCH_CHECK();
  lazy_flush_commit_kernel<<<ceil_div(n_texels, 256), 256, 0, stream>>>(last_step, n_texels, t);
  LMB_LAUNCH_CHECK();
  return 0;
}
