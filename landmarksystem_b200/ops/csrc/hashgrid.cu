// Multiresolution hash-grid encoding (Instant-NGP style), forward and backward.
//
// Level l: pos = x * scale_l + 0.5; the 8 corners of the enclosing cell are looked up in the level's
// table (dense index when the grid fits, XOR-of-primes spatial hash otherwise) and blended
// trilinearly.  The reference gets this op from tiny-cuda-nn (landmark/nerf_components/
// model_components/fields/encodings/hash_encoding.py:82-107).
//
// Work layout: one thread handles one sample and a group of kLevelGroup consecutive levels; blockIdx.y is the level
// group and varies slowest.  A warp is therefore 32 consecutive samples (neighbours along a ray) at the same levels:
//  * on the coarse levels neighbouring samples sit in the same cell, so their corner loads coalesce into a few
//    sectors, and in the backward their contributions are summed inside the warp (segmented over runs of equal cells)
//    before one lane per run touches memory;
//  * the tables of one level group (4 x 2^22 entries at most) are the only ones in flight while the grid sweeps the
//    samples, instead of all 16 levels competing for the L2;
//  * a thread's outputs are 4 levels x F features = one full 32-byte sector of the sample's row.
#include "hashgrid.cuh"

namespace lmb {

constexpr int kLevelGroup = 4;
// The backward sweeps two levels at a time: their fp32 gradient tables (2 x 2^22 entries x 8 bytes = 64 MB at the
// benchmark shape) stay resident in the 126 MB L2 while the grid walks the samples, so the reductions on the hashed
// levels complete in the L2 instead of fetching and writing back a DRAM sector each.  Measured on the Instant-NGP
// benchmark step (42 M samples, 16 levels): 105.6 ms with four levels per sweep, 91.5 ms with two, 92.1 ms with one.
constexpr int kBwdLevelGroup = 2;
constexpr int kWarpReduceMaxRes = 512;   // levels up to this resolution pre-reduce their gradients inside the warp

template <typename T, int F>
__device__ __forceinline__ void load_entry(const T* e, float* v) {
  if constexpr (sizeof(T) == 4 && F == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(e));
    v[0] = t.x; v[1] = t.y;
  } else if constexpr (sizeof(T) == 4 && F == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(e));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr (sizeof(T) == 2 && F == 2) {
    const unsigned u = __ldg(reinterpret_cast<const unsigned*>(e));
    const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
    v[0] = t.x; v[1] = t.y;
  } else if constexpr (sizeof(T) == 2 && F == 8) {
    const F8 t = load8(reinterpret_cast<const __nv_bfloat16*>(e));
#pragma unroll
    for (int f = 0; f < 8; ++f) v[f] = t.v[f];
  } else {
#pragma unroll
    for (int f = 0; f < F; ++f) v[f] = (float)e[f];
  }
}

// Entries a and b of an edge along x.  x enters the spatial hash with factor 1 and a dense index directly, so the two entries
// of every other edge are the halves of one aligned pair (a ^ b = 1): one request of twice the size instead of two.  131072-ray Instant-NGP
// step, with the steps of the backward's warp sums that add nothing left out: forward 3056 -> 2804 us, backward 5344 -> 4409 us.
template <typename T, int F>
__device__ __forceinline__ void load_edge(const T* tab, uint32_t a, uint32_t b, bool pairs, float* e0, float* e1) {
  if constexpr (F == 2) {
    if (pairs) {
      float lo[2], hi[2];
      const T* pair = tab + (long long)(a & ~1u) * 2;
      if constexpr (sizeof(T) == 2) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(pair));
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        lo[0] = x.x; lo[1] = x.y; hi[0] = y.x; hi[1] = y.y;
      } else {
        const float4 u = __ldg(reinterpret_cast<const float4*>(pair));
        lo[0] = u.x; lo[1] = u.y; hi[0] = u.z; hi[1] = u.w;
      }
      const bool odd = a & 1u;
      e0[0] = odd ? hi[0] : lo[0]; e0[1] = odd ? hi[1] : lo[1];
      e1[0] = odd ? lo[0] : hi[0]; e1[1] = odd ? lo[1] : hi[1];
      if ((a ^ b) != 1u) load_entry<T, F>(tab + (long long)b * F, e1);
      return;
    }
  }
  load_entry<T, F>(tab + (long long)a * F, e0);
  load_entry<T, F>(tab + (long long)b * F, e1);
}

template <typename T, typename OutT, int F>
__global__ void __launch_bounds__(256)
hashgrid_fwd_kernel(const float* __restrict__ x, long long n, const T* __restrict__ table, HashMeta m, bool pairs,
                    OutT* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int L = m.n_levels;
  const int l0 = blockIdx.y * kLevelGroup;
  const float xs[3] = {x[i * 3], x[i * 3 + 1], x[i * 3 + 2]};
  float acc[kLevelGroup][F];
#pragma unroll
  for (int g = 0; g < kLevelGroup; ++g) {
    const int l = l0 + g;
#pragma unroll
    for (int f = 0; f < F; ++f) acc[g][f] = 0.f;
    if (l >= L) continue;
    const float scale = m.scale[l];
    const LevelIndex index((uint32_t)m.res[l], (uint32_t)(m.offset[l + 1] - m.offset[l]));
    const T* tab = table + m.offset[l] * F;
    float w[3];
    uint32_t p0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float p = xs[d] * scale + 0.5f;
      const float fl = floorf(p);
      w[d] = p - fl;
      p0[d] = (uint32_t)max((int)fl, 0);
    }
#pragma unroll
    for (int c = 0; c < 8; c += 2) {                          // the two corners of an edge along x
      const uint32_t iy = min(p0[1] + ((c >> 1) & 1), index.res - 1), iz = min(p0[2] + ((c >> 2) & 1), index.res - 1);
      const uint32_t a = index(min(p0[0], index.res - 1), iy, iz), b = index(min(p0[0] + 1, index.res - 1), iy, iz);
      const float w0 = (1.f - w[0]) * ((c & 2) ? w[1] : 1.f - w[1]) * ((c & 4) ? w[2] : 1.f - w[2]);
      const float w1 = w[0] * ((c & 2) ? w[1] : 1.f - w[1]) * ((c & 4) ? w[2] : 1.f - w[2]);
      float e0[F], e1[F];
      load_edge<T, F>(tab, a, b, pairs, e0, e1);
#pragma unroll
      for (int f = 0; f < F; ++f) { acc[g][f] += w0 * e0[f]; acc[g][f] += w1 * e1[f]; }
    }
  }
  OutT* o = out + i * (long long)(L * F) + l0 * F;
  if (F == 2 && L % kLevelGroup == 0) {
    // 4 levels x 2 features: one 32-byte (fp32) or 16-byte (bf16) piece of the row, aligned because L*F is a multiple of 8
    if constexpr (sizeof(OutT) == 4) {
      reinterpret_cast<float4*>(o)[0] = make_float4(acc[0][0], acc[0][F > 1 ? 1 : 0], acc[1][0], acc[1][F > 1 ? 1 : 0]);
      reinterpret_cast<float4*>(o)[1] = make_float4(acc[2][0], acc[2][F > 1 ? 1 : 0], acc[3][0], acc[3][F > 1 ? 1 : 0]);
    } else {
      F8 v;
#pragma unroll
      for (int g = 0; g < kLevelGroup; ++g) { v.v[2 * g] = acc[g][0]; v.v[2 * g + 1] = acc[g][F > 1 ? 1 : 0]; }
      store8(reinterpret_cast<__nv_bfloat16*>(o), v);
    }
  } else {
#pragma unroll
    for (int g = 0; g < kLevelGroup; ++g)
      if (l0 + g < L) {
#pragma unroll
        for (int f = 0; f < F; ++f) o[g * F + f] = (OutT)acc[g][f];
      }
  }
}

template <int F>
__device__ __forceinline__ void red_entry(float* e, const float* v) {
  if constexpr (F == 2) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(e), "f"(v[0]), "f"(v[1]) : "memory");
  } else if constexpr (F == 4) {
    red_add_v4(e, v[0], v[1], v[2], v[3]);
  } else if constexpr (F == 8) {
    red_add_v4(e, v[0], v[1], v[2], v[3]);
    red_add_v4(e + 4, v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int f = 0; f < F; ++f) atomicAdd(e + f, v[f]);
  }
}

// Adds v0 and v1 to entries a and b of an edge along x; two features of an aligned pair travel as one 16-byte reduction.
template <int F>
__device__ __forceinline__ void red_edge(float* tab, uint32_t a, uint32_t b, bool pairs, const float* v0, const float* v1) {
  if constexpr (F == 2) {
    if (pairs && (a ^ b) == 1u) {
      const bool odd = a & 1u;
      red_add_v4(tab + (long long)(a & ~1u) * 2, odd ? v1[0] : v0[0], odd ? v1[1] : v0[1], odd ? v0[0] : v1[0], odd ? v0[1] : v1[1]);
      return;
    }
  }
  red_entry<F>(tab + (long long)a * F, v0);
  red_entry<F>(tab + (long long)b * F, v1);
}

template <typename GT, int F, int LG>
__global__ void __launch_bounds__(256)
hashgrid_bwd_kernel(const float* __restrict__ x, long long n, HashMeta m, bool pairs, const GT* __restrict__ dout,
                    float* __restrict__ grad) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  const int lane = threadIdx.x & 31;
  const int L = m.n_levels;
  const int l0 = blockIdx.y * LG;
  float xs[3] = {0.f, 0.f, 0.f};
  if (live) { xs[0] = x[i * 3]; xs[1] = x[i * 3 + 1]; xs[2] = x[i * 3 + 2]; }
#pragma unroll 1
  for (int g = 0; g < LG; ++g) {
    const int l = l0 + g;
    if (l >= L) break;                                      // uniform
    float gv[F];
    bool any = false;
    if (live) {
      const GT* gp = dout + i * (long long)(L * F) + l * F;
#pragma unroll
      for (int f = 0; f < F; ++f) { gv[f] = (float)gp[f]; any |= gv[f] != 0.f; }
    } else {
#pragma unroll
      for (int f = 0; f < F; ++f) gv[f] = 0.f;
    }
    const float scale = m.scale[l];
    const LevelIndex index((uint32_t)m.res[l], (uint32_t)(m.offset[l + 1] - m.offset[l]));
    float* tab = grad + m.offset[l] * F;
    float w[3];
    uint32_t p0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float p = xs[d] * scale + 0.5f;
      const float fl = floorf(p);
      w[d] = p - fl;
      p0[d] = (uint32_t)max((int)fl, 0);
    }
    if ((int)index.res <= kWarpReduceMaxRes) {
      // Runs of consecutive lanes in the same cell (res <= 512: the cell packs into 30 bits, and positions past the grid clamp to
      // the last cell in the key as they do in the index; a lane without a gradient gets a key of its own) are summed with a segmented suffix reduction; the first lane of a run writes.
      const uint32_t key = (live && any) ? (min(p0[0], 1023u) | (min(p0[1], 1023u) << 10) | (min(p0[2], 1023u) << 20))
                                          : (0xC0000000u | (uint32_t)lane);
      const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
      const bool head = lane == 0 || prev != key;
      const unsigned heads = __ballot_sync(0xffffffffu, head);
      const int seg = __popc(heads & (0xffffffffu >> (31 - lane)));
      bool take[5];
      // z[s]: somewhere a run goes on for more than 2^s lanes; without one the step adds nothing (warp-uniform)
      unsigned z[5];
      z[0] = ~heads; z[1] = z[0] & z[0] >> 1; z[2] = z[1] & z[1] >> 2; z[3] = z[2] & z[2] >> 4; z[4] = z[3] & z[3] >> 8;
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        const int other = __shfl_down_sync(0xffffffffu, seg, 1 << s);
        take[s] = (lane + (1 << s) < 32) && other == seg;
      }
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        float v[2][F];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float wt = (k ? w[0] : 1.f - w[0]) * ((c & 2) ? w[1] : 1.f - w[1]) * ((c & 4) ? w[2] : 1.f - w[2]);
#pragma unroll
          for (int f = 0; f < F; ++f) v[k][f] = wt * gv[f];
        }
#pragma unroll
        for (int s = 0; s < 5; ++s)
          if (z[s]) {
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
              for (int f = 0; f < F; ++f) {
                const float o = __shfl_down_sync(0xffffffffu, v[k][f], 1 << s);
                if (take[s]) v[k][f] += o;
              }
          }
        if (head && live && any) {
          const uint32_t iy = min(p0[1] + ((c >> 1) & 1), index.res - 1), iz = min(p0[2] + ((c >> 2) & 1), index.res - 1);
          red_edge<F>(tab, index(min(p0[0], index.res - 1), iy, iz), index(min(p0[0] + 1, index.res - 1), iy, iz), pairs, v[0], v[1]);
        }
      }
    } else if (live && any) {
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        const uint32_t iy = min(p0[1] + ((c >> 1) & 1), index.res - 1), iz = min(p0[2] + ((c >> 2) & 1), index.res - 1);
        float v[2][F];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float wt = (k ? w[0] : 1.f - w[0]) * ((c & 2) ? w[1] : 1.f - w[1]) * ((c & 4) ? w[2] : 1.f - w[2]);
#pragma unroll
          for (int f = 0; f < F; ++f) v[k][f] = wt * gv[f];
        }
        red_edge<F>(tab, index(min(p0[0], index.res - 1), iy, iz), index(min(p0[0] + 1, index.res - 1), iy, iz), pairs, v[0], v[1]);
      }
    }
  }
}

}  // namespace lmb

using namespace lmb;

#define LMB_DISPATCH_F(F_, ...)            \
  switch (F_) {                            \
    case 1: { constexpr int F = 1; __VA_ARGS__; break; } \
    case 2: { constexpr int F = 2; __VA_ARGS__; break; } \
    case 4: { constexpr int F = 4; __VA_ARGS__; break; } \
    case 8: { constexpr int F = 8; __VA_ARGS__; break; } \
    default: return (int)cudaErrorInvalidValue; \
  }

// Levels start at an even entry and the array on a pair of entries, so that an aligned pair never leaves its level.
static bool pairs_allowed(const HashMeta* meta, const void* base, size_t pair_bytes) {
  for (int l = 0; l <= meta->n_levels; ++l)
    if (meta->offset[l] & 1) return false;
  return (uintptr_t)base % pair_bytes == 0;
}

LMB_API int lmb_hashgrid_fwd(const float* x, long long n, const void* table, int table_dtype, const HashMeta* meta,
                             void* out, int out_dtype, cudaStream_t stream) {
  if (n <= 0) return 0;
  const dim3 blocks(ceil_div(n, 256), ceil_div(meta->n_levels, kLevelGroup));
  const bool pairs = pairs_allowed(meta, table, table_dtype == 0 ? 16 : 8);
  LMB_DISPATCH_F(meta->n_features, {
    if (table_dtype == 0 && out_dtype == 0)
      hashgrid_fwd_kernel<float, float, F><<<blocks, 256, 0, stream>>>(x, n, (const float*)table, *meta, pairs, (float*)out);
    else if (table_dtype == 1 && out_dtype == 0)
      hashgrid_fwd_kernel<__nv_bfloat16, float, F><<<blocks, 256, 0, stream>>>(x, n, (const __nv_bfloat16*)table, *meta, pairs, (float*)out);
    else if (table_dtype == 0 && out_dtype == 1)
      hashgrid_fwd_kernel<float, __nv_bfloat16, F><<<blocks, 256, 0, stream>>>(x, n, (const float*)table, *meta, pairs, (__nv_bfloat16*)out);
    else
      hashgrid_fwd_kernel<__nv_bfloat16, __nv_bfloat16, F><<<blocks, 256, 0, stream>>>(x, n, (const __nv_bfloat16*)table, *meta, pairs, (__nv_bfloat16*)out);
  });
  LMB_LAUNCH_CHECK();
  return 0;
}

LMB_API int lmb_hashgrid_bwd(const float* x, long long n, const HashMeta* meta, const void* dout, int dout_dtype,
                             float* grad, cudaStream_t stream) {
  if (n <= 0) return 0;
  const dim3 blocks(ceil_div(n, 256), ceil_div(meta->n_levels, kBwdLevelGroup));
  const bool pairs = pairs_allowed(meta, grad, 16);
  LMB_DISPATCH_F(meta->n_features, {
    if (dout_dtype == 0)
      hashgrid_bwd_kernel<float, F, kBwdLevelGroup><<<blocks, 256, 0, stream>>>(x, n, *meta, pairs, (const float*)dout, grad);
    else
      hashgrid_bwd_kernel<__nv_bfloat16, F, kBwdLevelGroup><<<blocks, 256, 0, stream>>>(x, n, *meta, pairs, (const __nv_bfloat16*)dout, grad);
  });
  LMB_LAUNCH_CHECK();
  return 0;
}
