// What the training forward (train.cu) and backward (train_bwd.cu) share: the
// shape of the field, the packed weights and the interpolation's weights.
#pragma once
#include "common.cuh"

namespace nsvf_train {

constexpr int kT = 256;
constexpr int kTile = 128;                 // samples per tile
constexpr int kHid = 128, kE = 32;
constexpr int kSMs = 152;

// packed FP32 weights: W_l transposed ([k][unit], l = 0..3), then W4 [4][128],
// b0..b3 [4][128], b4 [4]
__host__ __device__ constexpr int w_off(int l) { return l ? (kE + (l - 1) * kHid) * kHid : 0; }
constexpr int kW4Off = (kE + 3 * kHid) * kHid;
constexpr int kBiasOff = kW4Off + 4 * kHid;
constexpr int kB4Off = kBiasOff + 4 * kHid;
constexpr int kPacked = kB4Off + 4;

// w_k for corner k, multiplied in dimension order (interp.cu)
__device__ __forceinline__ float corner_weight(const float p[3], int k) {
  const float a = (k & 4) ? p[0] : 1.0f - p[0];
  const float b = (k & 2) ? p[1] : 1.0f - p[1];
  const float c = (k & 1) ? p[2] : 1.0f - p[2];
  return a * b * c;
}

inline bool bad_scene(int64_t ns, const int32_t *vox, const float *xyzd, int64_t n_vox,
                      int64_t n_keys, const float *centers, const int32_t *feats,
                      const float *values, const float *packed) {
  return ns < 0 || n_vox < 0 || n_keys < 0 ||
         (ns > 0 && (!vox || !xyzd || !centers || !feats || !values || !packed)) ||
         ((((uintptr_t)xyzd) | ((uintptr_t)values) | ((uintptr_t)packed)) & 15);
}

}  // namespace nsvf_train
