// Small perceptrons (at most 64 inputs, hidden layers of at most 64 units, relu between layers): forward and training
// backward with the activations of a row tile held in registers.
//
// The density and colour heads of the hash-grid models, the proposal networks and the anchor heads are this narrow
// (benchmarks/nerf/instant_ngp/instant_ngp.py:120-170 of the reference, which trains them through tiny-cuda-nn).  A layer of
// such a network is 0.5 MFLOP per 64 rows against 25 KB of row traffic, so the tensor pipe is not what bounds it: on the
// tcgen05 kernels (fused_mlp.cu, fused_mlp_bwd.cu) a layer is a hand-over MMA -> commit -> TMEM load -> conversion -> shared
// memory -> barrier, each several times longer than the tensor work of a 128 x 64 x 64 tile, and the backward kernel pads
// every layer to 128 columns and leaves one 128-thread block on an SM.  With warp-level MMAs the accumulator fragment of a
// layer IS the operand fragment of the next one, so a warp runs its 16 or 32 rows through the whole network without a
// barrier, and weights are the only shared-memory traffic.  The tcgen05 kernels stay for wider networks, where an operand
// tile no longer fits in registers.
//
// Rounding is that of the tcgen05 kernels: bf16 inputs, activations and back-propagated gradients, fp32 sums.
#include "fused_mlp.cuh"

namespace lmb {

constexpr int kHid = 64;                       // padded hidden width
constexpr int kHidPitch = kHid * 2 + 16;       // shared-memory rows end with 16 spare bytes: 8 rows of a matrix load hit all banks
__host__ __device__ constexpr int pitch_of(int cols) { return cols * 2 + 16; }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t pack2_relu(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// the halves of v whose counterpart in h (an activation after relu) is positive
__device__ __forceinline__ uint32_t where_positive(uint32_t v, uint32_t h) {
  return v & (((h & 0xFFFFu) ? 0xFFFFu : 0u) | ((h >> 16) ? 0xFFFF0000u : 0u));
}

// Per-lane offsets of the four 8x8 matrices of a matrix load over row-major storage.
//   frag : 16 x 16 operand A (rows x k), or with .trans the operand A^T of a product over rows
//   pair : operand B = W^T for 16 outputs and 16 k from W [outputs][k]; with .trans two 8-column tiles of B = W [k][columns]
__device__ __forceinline__ uint32_t off_frag(int lane, int pitch) { return ((lane >> 3 & 1) * 8 + (lane & 7)) * pitch + (lane >> 4) * 16; }
__device__ __forceinline__ uint32_t off_pair(int lane, int pitch) { return ((lane >> 4) * 8 + (lane & 7)) * pitch + (lane >> 3 & 1) * 16; }
__device__ __forceinline__ uint32_t off_rows(int lane, int pitch) { return lane * pitch; }      // 32 rows of one 8-column tile

// Weights of one layer from the packed blob [k / 8][blob_n][8] into row-major shared memory [n_pad][k_pad], zero beyond
__device__ __forceinline__ void stage_weights(const unsigned char* __restrict__ blob, int blob_n, int blob_k, unsigned char* s, int n_pad,
                                              int k_pad) {
  const int chunks = k_pad / 8, pitch = pitch_of(k_pad);
  for (int i = threadIdx.x; i < n_pad * chunks; i += blockDim.x) {
    const int n = i % n_pad, c = i / n_pad;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (n < blob_n && c * 8 < blob_k) v = __ldg(reinterpret_cast<const uint4*>(blob) + (size_t)c * blob_n + n);
    *reinterpret_cast<uint4*>(s + n * pitch + c * 16) = v;
  }
}

// 16 input rows of one warp into shared memory, zero beyond the tensor's rows and columns
template <int kRows>
__device__ __forceinline__ void stage_rows(const __nv_bfloat16* __restrict__ x, long long row0, long long n, int width, int k_pad,
                                           unsigned char* s) {
  const int chunks = k_pad / 8, pitch = pitch_of(k_pad);
#pragma unroll 4
  for (int i = threadIdx.x & 31; i < kRows * chunks; i += 32) {
    const int r = i / chunks, c = i % chunks;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (row0 + r < n && c * 8 < width) v = __ldg(reinterpret_cast<const uint4*>(x + (row0 + r) * width) + c);
    *reinterpret_cast<uint4*>(s + r * pitch + c * 16) = v;
  }
}

// One layer for M row tiles of 16: acc = a [.. x 16 KT] * W^T, all kHid outputs
template <int M, int KT>
__device__ __forceinline__ void layer64(float (&acc)[M][8][4], const uint32_t (&a)[M][KT][4], uint32_t w, int pitch, int lane) {
  const uint32_t at = w + off_pair(lane, pitch);
#pragma unroll
  for (int kt = 0; kt < KT; ++kt)
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      uint32_t b[4];
      ldsm4(b, at + np * 16 * pitch + kt * 32);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        mma_bf16(acc[m][2 * np], a[m][kt], b[0], b[1]);
        mma_bf16(acc[m][2 * np + 1], a[m][kt], b[2], b[3]);
      }
    }
}

template <int M>
__device__ __forceinline__ void init_acc(float (&acc)[M][8][4], const float* bias, int lane) {
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    const float lo = bias ? bias[nt * 8 + 2 * (lane & 3)] : 0.f, hi = bias ? bias[nt * 8 + 2 * (lane & 3) + 1] : 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) { acc[m][nt][0] = acc[m][nt][2] = lo; acc[m][nt][1] = acc[m][nt][3] = hi; }
  }
}

// relu and rounding: the accumulator fragment of 64 outputs as the A fragment of the next layer
template <int M>
__device__ __forceinline__ void relu_frag(uint32_t (&h)[M][4][4], const float (&acc)[M][8][4]) {
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      h[m][kt][0] = pack2_relu(acc[m][2 * kt][0], acc[m][2 * kt][1]);
      h[m][kt][1] = pack2_relu(acc[m][2 * kt][2], acc[m][2 * kt][3]);
      h[m][kt][2] = pack2_relu(acc[m][2 * kt + 1][0], acc[m][2 * kt + 1][1]);
      h[m][kt][3] = pack2_relu(acc[m][2 * kt + 1][2], acc[m][2 * kt + 1][3]);
    }
}

// ---- forward --------------------------------------------------------------------------------------------------
constexpr int kFwdWarps = 4, kFwdM = 2, kFwdRows = 16 * kFwdM;      // rows per warp and step

struct NarrowFwdLayout { int w1, w2, w3, bias, rows, bytes; };      // byte offsets in shared memory
__host__ __device__ inline NarrowFwdLayout narrow_fwd_layout(int k0, int layers, int n_last) {
  NarrowFwdLayout l;
  l.w1 = 0;
  l.w2 = l.w1 + kHid * pitch_of(k0);
  l.w3 = l.w2 + (layers == 3 ? kHid * kHidPitch : 0);
  l.bias = l.w3 + n_last * kHidPitch;
  l.rows = l.bias + (2 * kHid + n_last) * 4;
  l.bytes = l.rows + kFwdWarps * kFwdRows * pitch_of(k0);
  return l;
}

// Bound by the latency of loads and MMAs at 14 warps an SM (2 Mi rows of 64 inputs: L1 at 59 % of its throughput, DRAM at 26 %,
// a third of the issue slots taken).  131072-ray Instant-NGP step: the two
// heads 2079 -> 1001 us; 800 x 800 frame 7625 -> 3887 us; the three anchor heads of a 400 k frame 225 -> 76 us.
template <int KT0>
__global__ void __launch_bounds__(kFwdWarps * 32, 4)
narrow_fwd_kernel(const __nv_bfloat16* __restrict__ x, const unsigned char* __restrict__ blob, MLPSpec spec,
                  const int* __restrict__ count_ptr, long long max_rows, float* __restrict__ out, int out_stride) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int K0 = KT0 * 16;
  const int layers = spec.n_layers, last = layers - 1, n_last = spec.N[last];
  const NarrowFwdLayout at = narrow_fwd_layout(K0, layers, n_last);
  const long long n = resolve_count(count_ptr, max_rows);
  if ((long long)blockIdx.x * kFwdWarps * kFwdRows >= n) return;
  stage_weights(blob + spec.w_off[0], spec.N[0], spec.K[0], smem + at.w1, kHid, K0);
  if (layers == 3) stage_weights(blob + spec.w_off[1], spec.N[1], spec.K[1], smem + at.w2, kHid, kHid);
  stage_weights(blob + spec.w_off[last], n_last, spec.K[last], smem + at.w3, n_last, kHid);
  float* bias = reinterpret_cast<float*>(smem + at.bias);
  for (int i = threadIdx.x; i < 2 * kHid + n_last; i += blockDim.x) {
    const int l = i < kHid ? 0 : (i < 2 * kHid ? 1 : last), c = i < kHid ? i : (i < 2 * kHid ? i - kHid : i - 2 * kHid);
    bias[i] = spec.b_off[l] >= 0 && c < spec.N[l] ? reinterpret_cast<const float*>(blob + spec.b_off[l])[c] : 0.f;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* rows = smem + at.rows + warp * kFwdRows * pitch_of(K0);
  const uint32_t base = tc05::smem_u32(smem), rows_u = tc05::smem_u32(rows);
  const int act = spec.act[last], out_dim = spec.out_dim;
  const bool pairs = (out_stride & 1) == 0 && (uintptr_t)out % 8 == 0;
  const long long step = (long long)gridDim.x * kFwdWarps * kFwdRows;
  for (long long row0 = ((long long)blockIdx.x * kFwdWarps + warp) * kFwdRows; row0 < n; row0 += step) {
    __syncwarp();
    stage_rows<kFwdRows>(x, row0, n, spec.in_width, K0, rows);
    __syncwarp();
    uint32_t h[kFwdM][4][4];
    {
      uint32_t a[kFwdM][KT0][4];
#pragma unroll
      for (int m = 0; m < kFwdM; ++m)
#pragma unroll
        for (int kt = 0; kt < KT0; ++kt) ldsm4(a[m][kt], rows_u + off_frag(lane, pitch_of(K0)) + m * 16 * pitch_of(K0) + kt * 32);
      float acc[kFwdM][8][4];
      init_acc<kFwdM>(acc, bias, lane);
      layer64<kFwdM, KT0>(acc, a, base + at.w1, pitch_of(K0), lane);
      relu_frag<kFwdM>(h, acc);
    }
    if (layers == 3) {
      float acc[kFwdM][8][4];
      init_acc<kFwdM>(acc, bias + kHid, lane);
      layer64<kFwdM, 4>(acc, h, base + at.w2, kHidPitch, lane);
      relu_frag<kFwdM>(h, acc);
    }
    for (int n0 = 0; n0 < n_last; n0 += 16) {
      float o[kFwdM][2][4];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float lo = bias[2 * kHid + n0 + t * 8 + 2 * (lane & 3)], hi = bias[2 * kHid + n0 + t * 8 + 2 * (lane & 3) + 1];
#pragma unroll
        for (int m = 0; m < kFwdM; ++m) { o[m][t][0] = o[m][t][2] = lo; o[m][t][1] = o[m][t][3] = hi; }
      }
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        uint32_t b[4];
        ldsm4(b, base + at.w3 + off_pair(lane, kHidPitch) + n0 * kHidPitch + kt * 32);
#pragma unroll
        for (int m = 0; m < kFwdM; ++m) { mma_bf16(o[m][0], h[m][kt], b[0], b[1]); mma_bf16(o[m][1], h[m][kt], b[2], b[3]); }
      }
#pragma unroll
      for (int m = 0; m < kFwdM; ++m)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const long long row = row0 + m * 16 + half * 8 + (lane >> 2);
          if (row >= n) continue;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int c = n0 + t * 8 + 2 * (lane & 3);
            float* p = out + row * out_stride + c;
            const float lo = apply_act(o[m][t][2 * half], act), hi = apply_act(o[m][t][2 * half + 1], act);
            if (c + 1 < out_dim && pairs) *reinterpret_cast<float2*>(p) = make_float2(lo, hi);
            else {
              if (c < out_dim) p[0] = lo;
              if (c + 1 < out_dim) p[1] = hi;
            }
          }
        }
    }
  }
}

// ---- backward --------------------------------------------------------------------------------------------------
constexpr int kBwdWarps = 8, kBwdTile = kBwdWarps * 16;             // a warp owns 16 rows of the block's tile
constexpr int kOutPitch = 16 * 2 + 16;

struct NarrowBwdLayout { int w1, w2, w3, x, h1, h2, dz1, dz3, bytes; };
__host__ __device__ inline NarrowBwdLayout narrow_bwd_layout(int k0, bool three) {
  NarrowBwdLayout l;
  l.w1 = 0;
  l.w2 = l.w1 + kHid * pitch_of(k0);
  l.w3 = l.w2 + (three ? kHid * kHidPitch : 0);
  l.x = l.w3 + 16 * kHidPitch;
  l.h1 = l.x + kBwdTile * pitch_of(k0);
  l.h2 = l.h1 + kBwdTile * kHidPitch;                               // h2, later dz2
  l.dz1 = l.h2 + (three ? kBwdTile * kHidPitch : 0);
  l.dz3 = l.dz1 + kBwdTile * kHidPitch;
  l.bytes = l.dz3 + kBwdTile * kOutPitch;
  return l;
}

__device__ __forceinline__ void store_frag(unsigned char* s, int pitch, int kt, const uint32_t (&f)[4], int lane) {
  unsigned char* p = s + (lane >> 2) * pitch + kt * 32 + (lane & 3) * 4;
  *reinterpret_cast<uint32_t*>(p) = f[0];
  *reinterpret_cast<uint32_t*>(p + 8 * pitch) = f[1];
  *reinterpret_cast<uint32_t*>(p + 16) = f[2];
  *reinterpret_cast<uint32_t*>(p + 8 * pitch + 16) = f[3];
}

// acc [16 x 8 NT] += dz[:, 16 columns]^T * h[:, 8 NT columns] over the tile's rows
template <int NT>
__device__ __forceinline__ void wgrad(float (&acc)[NT][4], uint32_t dz, int dz_pitch, uint32_t h, int h_pitch, int lane) {
  const uint32_t a_at = dz + off_pair(lane, dz_pitch), b_at = h + off_rows(lane, h_pitch);
#pragma unroll
  for (int r = 0; r < kBwdTile; r += 32) {
    uint32_t a0[4], a1[4];
    ldsm4t(a0, a_at + r * dz_pitch);
    ldsm4t(a1, a_at + (r + 16) * dz_pitch);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      uint32_t b[4];
      ldsm4t(b, b_at + r * h_pitch + t * 16);
      mma_bf16(acc[t], a0, b[0], b[1]);
      mma_bf16(acc[t], a1, b[2], b[3]);
    }
  }
}

// gradient of the layer's input: acc [16 x 8 NT] = dz [16 x 16 KT] * W, W [outputs][columns]
template <int KT, int NT>
__device__ __forceinline__ void dgrad(float (&acc)[NT][4], const uint32_t (&dz)[KT][4], uint32_t w, int pitch, int lane) {
  const uint32_t at = w + off_frag(lane, pitch);
#pragma unroll
  for (int t = 0; t < NT; ++t) { acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f; }
#pragma unroll
  for (int kt = 0; kt < KT; ++kt)
#pragma unroll
    for (int np = 0; np < NT / 2; ++np) {
      uint32_t b[4];
      ldsm4t(b, at + kt * 16 * pitch + np * 32);
      mma_bf16(acc[2 * np], dz[kt], b[0], b[1]);
      mma_bf16(acc[2 * np + 1], dz[kt], b[2], b[3]);
    }
}

// masked, rounded hidden gradient as an A fragment
__device__ __forceinline__ void masked_frag(uint32_t (&dz)[4][4], const float (&acc)[8][4], const uint32_t (&h)[4][4]) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    dz[kt][0] = where_positive(pack2(acc[2 * kt][0], acc[2 * kt][1]), h[kt][0]);
    dz[kt][1] = where_positive(pack2(acc[2 * kt][2], acc[2 * kt][3]), h[kt][1]);
    dz[kt][2] = where_positive(pack2(acc[2 * kt + 1][0], acc[2 * kt + 1][1]), h[kt][2]);
    dz[kt][3] = where_positive(pack2(acc[2 * kt + 1][2], acc[2 * kt + 1][3]), h[kt][3]);
  }
}

// Four 8-column tiles of a fragment row, a word (two columns) of each in every lane of a quad -> the whole tile of the lane's
// number in the quad, so that a row leaves in 16-byte pieces that are neighbours (10 M rows of 64 inputs, three layers: 2868 -> 2517 us
// together with the output gradient in pairs).
__device__ __forceinline__ uint4 quad_transpose(const uint32_t (&w)[4], int lane) {
  const bool high = lane & 2, odd = lane & 1;
  const uint32_t o0 = __shfl_xor_sync(0xffffffffu, high ? w[0] : w[2], 2), o1 = __shfl_xor_sync(0xffffffffu, high ? w[1] : w[3], 2);
  const uint32_t s0 = high ? w[2] : w[0], s1 = high ? w[3] : w[1];           // two tiles: own words, and those of the lane two away
  const uint32_t r = __shfl_xor_sync(0xffffffffu, odd ? s0 : s1, 1), ro = __shfl_xor_sync(0xffffffffu, odd ? o0 : o1, 1);
  const uint32_t own = odd ? s1 : s0, other = odd ? o1 : o0;
  const uint2 near = odd ? make_uint2(r, own) : make_uint2(own, r), far = odd ? make_uint2(ro, other) : make_uint2(other, ro);
  return high ? make_uint4(far.x, far.y, near.x, near.y) : make_uint4(near.x, near.y, far.x, far.y);
}

template <int NT>
__device__ __forceinline__ void flush_wgrad(float* __restrict__ g, int row_pitch, int m0, int n0, const float (&acc)[NT][4], int lane) {
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float* p = g + (m0 + half * 8 + (lane >> 2)) * row_pitch + n0 + t * 8 + 2 * (lane & 3);
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(acc[t][2 * half]), "f"(acc[t][2 * half + 1]) : "memory");
    }
}

// Recompute, data gradients and weight gradients of a 128-row tile.  A warp takes its 16 rows forward and back in registers;
// x, the activations and the back-propagated gradients also go to shared memory, where all warps read them for the weight
// gradients (a product over the tile's rows): warp w owns 16 outputs (w % 4) and half of the inputs (w / 4) of the hidden
// layers and 8 inputs of the output layer, 28 - 36 accumulators a thread that stay in registers across tiles and leave once
// per block.  dz2 takes the place of h2 once the output layer's gradient has used it, so that two blocks fit on an SM.
// Bound by shared-memory operand loads, with 16 warps per SM in flight (2 Mi rows, three layers: L1 at 82 % of its throughput, a
// quarter of the issue slots taken, DRAM at 12 %).  131072-ray Instant-NGP step: the
// two heads 7822 -> 3456 us; 16384-ray Nerfacto step 615 -> 284 us.
template <int KT0, bool kThree>
__global__ void __launch_bounds__(kBwdWarps * 32, 2)
narrow_bwd_kernel(const __nv_bfloat16* __restrict__ x, int x_width, const unsigned char* __restrict__ blob, MLPSpec spec,
                  const int* __restrict__ count_ptr, long long max_rows, const float* __restrict__ dout, int dout_stride,
                  __nv_bfloat16* __restrict__ dx, float* __restrict__ gbuf) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int K0 = KT0 * 16, kPitch0 = pitch_of(K0);
  const NarrowBwdLayout at = narrow_bwd_layout(K0, kThree);
  const long long n = resolve_count(count_ptr, max_rows);
  if ((long long)blockIdx.x * kBwdTile >= n) return;
  stage_weights(blob + spec.w_off[0], spec.N[0], spec.K[0], smem + at.w1, kHid, K0);
  if (kThree) stage_weights(blob + spec.w_off[1], spec.N[1], spec.K[1], smem + at.w2, kHid, kHid);
  stage_weights(blob + spec.w_off[2], 16, spec.K[2], smem + at.w3, 16, kHid);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = tc05::smem_u32(smem);
  const uint32_t w1 = base + at.w1, w2 = base + at.w2, w3 = base + at.w3;
  unsigned char *sx = smem + at.x + warp * 16 * kPitch0, *sh1 = smem + at.h1 + warp * 16 * kHidPitch,
                *sh2 = smem + at.h2 + warp * 16 * kHidPitch, *sdz1 = smem + at.dz1 + warp * 16 * kHidPitch,
                *sdz3 = smem + at.dz3 + warp * 16 * kOutPitch;
  const int m0 = (warp & 3) * 16, half = warp >> 2;
  const bool sigmoid = spec.act[2] == ACT_SIGMOID;
  const bool whole = (uintptr_t)dx % 16 == 0 && x_width % 8 == 0, pairs = (uintptr_t)dout % 8 == 0 && dout_stride % 2 == 0;
  const int out_dim = spec.out_dim;
  float g1[KT0][4], g2[4][4], g3[1][4];
#pragma unroll
  for (int t = 0; t < KT0; ++t) { g1[t][0] = g1[t][1] = g1[t][2] = g1[t][3] = 0.f; }
#pragma unroll
  for (int t = 0; t < 4; ++t) { g2[t][0] = g2[t][1] = g2[t][2] = g2[t][3] = 0.f; }
  g3[0][0] = g3[0][1] = g3[0][2] = g3[0][3] = 0.f;

  for (long long tile0 = (long long)blockIdx.x * kBwdTile; tile0 < n; tile0 += (long long)gridDim.x * kBwdTile) {
    const long long row0 = tile0 + warp * 16;
    stage_rows<16>(x, row0, n, x_width, K0, sx);
    float d[2][4];                                                  // dout, then dz of the output layer (fragment of 16 columns)
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const long long row = row0 + (k >> 1) * 8 + (lane >> 2);
        const int c = t * 8 + 2 * (lane & 3);
        const float* g = dout + row * dout_stride + c;
        if (pairs && row < n && c + 1 < out_dim) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(g));
          d[t][k] = v.x; d[t][k + 1] = v.y;
        } else {
          d[t][k] = row < n && c < out_dim ? __ldg(g) : 0.f;
          d[t][k + 1] = row < n && c + 1 < out_dim ? __ldg(g + 1) : 0.f;
        }
      }
    __syncwarp();
    uint32_t h1[1][4][4], h2[1][4][4];
    {
      uint32_t a[1][KT0][4];
#pragma unroll
      for (int kt = 0; kt < KT0; ++kt) ldsm4(a[0][kt], tc05::smem_u32(sx) + off_frag(lane, kPitch0) + kt * 32);
      float acc[1][8][4];
      init_acc<1>(acc, nullptr, lane);
      layer64<1, KT0>(acc, a, w1, kPitch0, lane);
      relu_frag<1>(h1, acc);
    }
    if (kThree) {
      float acc[1][8][4];
      init_acc<1>(acc, nullptr, lane);
      layer64<1, 4>(acc, h1, w2, kHidPitch, lane);
      relu_frag<1>(h2, acc);
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) store_frag(sh2, kHidPitch, kt, h2[0][kt], lane);
    }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) store_frag(sh1, kHidPitch, kt, h1[0][kt], lane);
    if (sigmoid) {
      float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        uint32_t b[4];
        ldsm4(b, w3 + off_pair(lane, kHidPitch) + kt * 32);
        mma_bf16(o[0], kThree ? h2[0][kt] : h1[0][kt], b[0], b[1]);
        mma_bf16(o[1], kThree ? h2[0][kt] : h1[0][kt], b[2], b[3]);
      }
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float s = apply_act(o[t][k], ACT_SIGMOID); d[t][k] *= s * (1.f - s); }
    }
    uint32_t dz3[1][4] = {{pack2(d[0][0], d[0][1]), pack2(d[0][2], d[0][3]), pack2(d[1][0], d[1][1]), pack2(d[1][2], d[1][3])}};
    store_frag(sdz3, kOutPitch, 0, dz3[0], lane);
    uint32_t dz[4][4];                                              // dz2 (three layers) or dz1
    {
      float acc[8][4];
      dgrad<1, 8>(acc, dz3, w3, kHidPitch, lane);
      masked_frag(dz, acc, kThree ? h2[0] : h1[0]);
    }
    if (kThree) {
      __syncthreads();
      wgrad<1>(g3, base + at.dz3, kOutPitch, base + at.h2 + warp * 16, kHidPitch, lane);
      __syncthreads();
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) store_frag(sh2, kHidPitch, kt, dz[kt], lane);
      float acc[8][4];
      dgrad<4, 8>(acc, dz, w2, kHidPitch, lane);
      masked_frag(dz, acc, h1[0]);
    }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) store_frag(sdz1, kHidPitch, kt, dz[kt], lane);
    {
      float acc[2 * KT0][4];
      dgrad<4, 2 * KT0>(acc, dz, w1, kPitch0, lane);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long row = row0 + h * 8 + (lane >> 2);
        int done = 0;                                                // tiles that left as whole pieces
        if (KT0 >= 2 && whole) {
#pragma unroll
          for (int t = 0; t + 4 <= 2 * KT0; t += 4) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = pack2(acc[t + k][2 * h], acc[t + k][2 * h + 1]);
            const uint4 piece = quad_transpose(w, lane);
            const int c = (t + (lane & 3)) * 8;
            if (row < n && c < x_width) *reinterpret_cast<uint4*>(dx + row * x_width + c) = piece;
          }
          done = 2 * KT0 / 4 * 4;
        }
#pragma unroll
        for (int t = 0; t < 2 * KT0; ++t) {
          const int c = t * 8 + 2 * (lane & 3);
          if (t >= done && row < n && c < x_width)
            *reinterpret_cast<uint32_t*>(dx + row * x_width + c) = pack2(acc[t][2 * h], acc[t][2 * h + 1]);
        }
      }
    }
    __syncthreads();
    if (kThree) wgrad<4>(g2, base + at.h2 + m0 * 2, kHidPitch, base + at.h1 + half * 64, kHidPitch, lane);
    else wgrad<1>(g3, base + at.dz3, kOutPitch, base + at.h1 + warp * 16, kHidPitch, lane);
    wgrad<KT0>(g1, base + at.dz1 + m0 * 2, kHidPitch, base + at.x + half * K0, kPitch0, lane);
    __syncthreads();
  }
  flush_wgrad<KT0>(gbuf + kG_DW1, 160, m0, half * (K0 / 2), g1, lane);
  if (kThree) flush_wgrad<4>(gbuf + kG_DW2, 144, m0, half * 32, g2, lane);
  // the output layer's gradient is kept input-major
#pragma unroll
  for (int k = 0; k < 4; ++k)
    atomicAdd(gbuf + kG_DW3T + (warp * 8 + 2 * (lane & 3) + (k & 1)) * 16 + (k >> 1) * 8 + (lane >> 2), g3[0][k]);
}

// ---- dispatch --------------------------------------------------------------------------------------------------
static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int KT0>
static int launch_fwd(const void* x, const int* count_ptr, long long max_rows, const void* blob, const MLPSpec& s, float* out,
                      int out_stride, cudaStream_t stream) {
  const int smem = narrow_fwd_layout(KT0 * 16, s.n_layers, s.N[s.n_layers - 1]).bytes;
  LMB_CUDA_TRY(cudaFuncSetAttribute(narrow_fwd_kernel<KT0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const long long tiles = (max_rows + kFwdWarps * kFwdRows - 1) / (kFwdWarps * kFwdRows), cap = 4LL * sm_count();
  narrow_fwd_kernel<KT0><<<(int)(tiles < cap ? tiles : cap), kFwdWarps * 32, smem, stream>>>(
      (const __nv_bfloat16*)x, (const unsigned char*)blob, s, count_ptr, max_rows, out, out_stride);
  LMB_LAUNCH_CHECK();
  return 0;
}

template <int KT0>
static int launch_bwd(const void* x, int x_width, const int* count_ptr, long long max_rows, const void* blob, const MLPSpec& s,
                      const float* dout, int dout_stride, void* dx, float* gbuf, cudaStream_t stream) {
  const bool three = s.K[1] != 0;
  const auto kernel = three ? narrow_bwd_kernel<KT0, true> : narrow_bwd_kernel<KT0, false>;
  const int smem = narrow_bwd_layout(KT0 * 16, three).bytes;
  LMB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const long long tiles = (max_rows + kBwdTile - 1) / kBwdTile, cap = 2LL * sm_count();
  kernel<<<(int)(tiles < cap ? tiles : cap), kBwdWarps * 32, smem, stream>>>((const __nv_bfloat16*)x, x_width, (const unsigned char*)blob,
                                                                            s, count_ptr, max_rows, dout, dout_stride,
                                                                            (__nv_bfloat16*)dx, gbuf);
  LMB_LAUNCH_CHECK();
  return 0;
}

// Two or three layers, at most 64 inputs and hidden units, relu in between, nothing folded into the weights; rows on 16 bytes.
bool narrow_fwd_supported(const void* x, const MLPSpec& s) {
  if (s.n_layers < 2 || s.n_layers > 3 || s.pe_stage || s.bias_in_gemm || s.K[0] > 64 || s.in_width > s.K[0] || (uintptr_t)x % 16)
    return false;
  for (int l = 0; l + 1 < s.n_layers; ++l)
    if (s.N[l] > kHid || s.K[l + 1] > kHid || s.act[l] != ACT_RELU) return false;
  return true;
}

int narrow_fwd(const void* x, const int* count_ptr, long long max_rows, const void* blob, const MLPSpec& s, float* out, int out_stride,
               cudaStream_t stream) {
  const auto run = s.K[0] <= 16 ? launch_fwd<1> : s.K[0] <= 32 ? launch_fwd<2> : s.K[0] <= 48 ? launch_fwd<3> : launch_fwd<4>;
  return run(x, count_ptr, max_rows, blob, s, out, out_stride, stream);
}

// No layer has a bias (bits 0 - 2 of bias_in_gemm), hidden units and input columns at most 64.
bool narrow_bwd_supported(const void* x, const void* dx, int x_width, const MLPSpec& s) {
  return (s.bias_in_gemm & 7) == 7 && s.hidden_cols > 0 && s.hidden_cols <= kHid && x_width <= 64 && (uintptr_t)x % 16 == 0 &&
         (uintptr_t)dx % 4 == 0;
}

int narrow_bwd(const void* x, int x_width, const int* count_ptr, long long max_rows, const void* blob, const MLPSpec& s,
               const float* dout, int dout_stride, void* dx, float* gbuf, cudaStream_t stream) {
  const auto run = x_width <= 16 ? launch_bwd<1> : x_width <= 32 ? launch_bwd<2> : x_width <= 48 ? launch_bwd<3> : launch_bwd<4>;
  return run(x, x_width, count_ptr, max_rows, blob, s, dout, dout_stride, dx, gbuf, stream);
}

}  // namespace lmb
