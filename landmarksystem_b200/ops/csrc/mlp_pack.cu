// Packing of a small network's weights into the device blob that the fused perceptron kernels read: fp32 [N, K] matrices to
// bf16 [K_pad / 8][N_pad][8] with zero padding, biases to fp32 [N_pad] and, where the layer wants it, into one column of its
// weights.
//
// An optimiser step changes the weights, so a training step packs every network again.  As tensor operations that was eight
// launches per layer (70 of the 187 launches of an Instant-NGP step, 40 of 116 in a recorded GridNeRF step); one kernel moves
// the 4 - 200 KB of a network at once.  Bound by its launch: GridNeRF step
// 1931 -> 1899 us (115 -> 91 launches); with the row form of the samples a 4096-ray Instant-NGP step 4162 -> 2965 us (187 ->
// 111 launches), and with the proposal kernels a Nerfacto step 6133 -> 5300 us (302 -> 250).
#include "common.cuh"

namespace lmb {

constexpr int kPackLayers = 5;

struct PackLayer {
  const float* w;        // [n, k], or null for the identity
  const float* b;        // [n] or null
  int n, k, n_pad, k_pad;
  int w_off, b_off;      // bytes; b_off < 0: no bias block
  int bias_col;          // column of the padded weights that holds the bias too, or -1
};

struct PackNet { PackLayer layer[kPackLayers]; int n_layers; };

__global__ void __launch_bounds__(256)
mlp_pack_kernel(PackNet net, unsigned char* __restrict__ blob) {
  int i = blockIdx.x * 256 + threadIdx.x;                              // one 16-byte piece
  for (int l = 0; l < net.n_layers; ++l) {
    const PackLayer& p = net.layer[l];
    const int pieces = p.n_pad * p.k_pad / 8;
    if (i < pieces) {
      const int n = i % p.n_pad, k0 = i / p.n_pad * 8;
      F8 v;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + j;
        float x = 0.f;
        if (p.w == nullptr) x = n == k ? 1.f : 0.f;
        else if (n < p.n && k < p.k) x = p.w[(long long)n * p.k + k];
        else if (k == p.bias_col && n < p.n && p.b != nullptr) x = p.b[n];
        v.v[j] = x;
      }
      store8(reinterpret_cast<__nv_bfloat16*>(blob + p.w_off) + (long long)i * 8, v);
      return;
    }
    i -= pieces;
    if (p.b_off < 0) continue;
    if (i < p.n_pad / 4) {
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = p.b != nullptr && 4 * i + j < p.n ? p.b[4 * i + j] : 0.f;
      reinterpret_cast<float4*>(blob + p.b_off)[i] = make_float4(x[0], x[1], x[2], x[3]);
      return;
    }
    i -= p.n_pad / 4;
  }
}

}  // namespace lmb

using namespace lmb;

// blob: 16-byte aligned, offsets multiples of 16, padded widths multiples of 16
LMB_API int lmb_mlp_pack(const PackNet* net, void* blob, cudaStream_t stream) {
  if (net->n_layers < 1 || net->n_layers > kPackLayers) return (int)cudaErrorInvalidValue;
  long long pieces = 0;
  for (int l = 0; l < net->n_layers; ++l) {
    const PackLayer& p = net->layer[l];
    if (p.n_pad % 16 || p.k_pad % 16 || p.w_off % 16 || p.n > p.n_pad || p.k > p.k_pad) return (int)cudaErrorInvalidValue;
    pieces += (long long)p.n_pad * p.k_pad / 8 + (p.b_off >= 0 ? p.n_pad / 4 : 0);
  }
  mlp_pack_kernel<<<ceil_div(pieces, 256), 256, 0, stream>>>(*net, (unsigned char*)blob);
  LMB_LAUNCH_CHECK();
  return 0;
}
