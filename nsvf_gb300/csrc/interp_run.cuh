// Trilinear interpolation of 32 channels over runs of samples: the corner
// weights and what a group of 8 lanes knows about its 4 consecutive samples
// (interp.cu, train_bwd.cu).
#pragma once
#include "common.cuh"

namespace nsvf_interp {

// w_k for corner k from p (q_kd in {0,1}: p*q + (1-p)*(1-q) reduces to p or
// 1-p exactly), multiplied in dimension order like torch's prod.
__device__ __forceinline__ float corner_w(const float p[3], int k) {
  float a = (k & 4) ? p[0] : 1.0f - p[0];
  float b = (k & 2) ? p[1] : 1.0f - p[1];
  float c = (k & 1) ? p[2] : 1.0f - p[2];
  return a * b * c;
}

constexpr int kLanes = 8, kRun = 4, kRunBlock = 128;

template <typename FeatT>
struct Group {
  int64_t v[kRun];          // voxel of each sample, -1 where there is none
  int key[kRun];            // this lane's corner of it, -1 where it is out of range
  float mine[3];            // trilinear coordinates of sample (lane & 3)

  // XS: floats between the positions
  template <int XS, typename IdxT>
  __device__ __forceinline__ void load(int64_t s0, int64_t ns, float voxel_size, int64_t n_vox,
                                       int64_t n_keys, const IdxT *__restrict__ sidx,
                                       const float *__restrict__ xyz,
                                       const float *__restrict__ centers,
                                       const FeatT *__restrict__ feats, int lane, int32_t *err) {
    const int64_t s = s0 + (lane & (kRun - 1));
    int64_t my = -1;
    mine[0] = mine[1] = mine[2] = 0.0f;
    if (s < ns) {
      my = (int64_t)sidx[s];
      if (my < 0 || my >= n_vox) {
        if (err) atomicOr(err, 4);
        my = -1;
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          mine[d] = (xyz[s * XS + d] - centers[my * 3 + d]) / voxel_size + 0.5f;
      }
    }
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
      v[i] = __shfl_sync(0xffffffffu, my, i, kLanes);
      if (i > 0 && v[i] == v[i - 1]) {
        key[i] = key[i - 1];
        continue;
      }
      key[i] = -1;
      if (v[i] < 0) continue;
      const int64_t k = (int64_t)feats[v[i] * 8 + lane];
      if (k >= 0 && k < n_keys) key[i] = (int)k;
      else if (err) atomicOr(err, 4);
    }
  }
  __device__ __forceinline__ bool change(int i) const { return i == 0 || v[i] != v[i - 1]; }
  __device__ __forceinline__ void coords(int i, float (&p)[3]) const {
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d] = __shfl_sync(0xffffffffu, mine[d], i, kLanes);
  }
};

}  // namespace nsvf_interp
