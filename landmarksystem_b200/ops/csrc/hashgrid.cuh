// Level layout and entry index of the multiresolution hash grid, shared by the kernels that look entries up.
#pragma once
#include "common.cuh"

namespace lmb {

struct HashMeta {
  float scale[32];
  int res[32];
  long long offset[33];
  int n_levels, n_features;
};

struct LevelIndex {
  uint32_t res, entries, mask;
  bool dense, pow2;
  __device__ __forceinline__ LevelIndex(uint32_t res_, uint32_t entries_) : res(res_), entries(entries_) {
    // dense when res^3 fits (res <= 1625 keeps res^3 inside 32 bits; larger grids always hash)
    dense = res <= 1625u && res * res * res <= entries;
    pow2 = (entries & (entries - 1u)) == 0u;
    mask = entries - 1u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t ix, uint32_t iy, uint32_t iz) const {
    if (dense) return ix + iy * res + iz * res * res;
    const uint32_t h = (ix * 1u) ^ (iy * 2654435761u) ^ (iz * 805459861u);
    return pow2 ? (h & mask) : (h % entries);
  }
};

}  // namespace lmb
