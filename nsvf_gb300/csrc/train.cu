// The forward of a training batch on compacted samples: FP32 interpolation and
// the 4 x 128 field (backward: train_bwd.cu), and the FP32 stage of pruning.
//
// Reference: SparseVoxelEncoder.forward (fairnr/modules/encoder.py:558-592),
// the field and VolumeRenderer.forward_chunk (fairnr/modules/renderer.py:
// 94-126) under autograd.
//
// Why a kernel of its own: the field's gradient is discontinuous where a
// pre-activation changes sign, so the forward has to keep FP32 and its order
// (one fused multiply-add chain over k = 0..K-1 from zero, then the bias:
// the bits of an FP32 SIMT GEMM with a bias epilogue), which leaves the
// tensor cores out. The bound is the FP32 pipe: 53,760 FMAs a sample. A chain
// of library GEMMs runs it at about 30 TFLOP/s and moves every activation
// through memory once per elementwise operation; here a tile of 128 samples
// goes through all layers in shared memory (1.40 M samples: 2.92 ms, 51
// TFLOP/s).
//
// field_train_kernel<MODE>, 256 threads, two blocks per SM (while one gathers
// or waits for weights, the other computes):
//   * activations [unit][sample] in shared memory (64 KB), each thread an 8 x
//     8 block of (unit, sample) accumulators, two samples per fma.rn.f32x2;
//   * the weights stream through three 8 KB stages by cp.async, in one
//     packed buffer that holds them in the order in which they are used, so a
//     stage is 2,048 consecutive floats and the next layer's weights arrive
//     during an epilogue;
//   * rows of 16-byte groups are XOR-swizzled by act_swz(row), so that the
//     epilogue's stores (8 rows, 4 apart), the GEMM's loads (one row) and the
//     head's loads are all free of bank conflicts.
// For a backward (kForwardSigns) it also writes the sign of every
// pre-activation, 64 bytes a sample: the backward recomputes activations to
// FP32 accuracy, but not to these bits.
#include "train_common.cuh"

using namespace nsvf_train;

namespace {

constexpr int kStages = 3;
constexpr int kStage = 2048;               // floats per weight stage
constexpr int kWStages = kW4Off / kStage;  // 26
constexpr int kBlocks = 2 * kSMs;          // two per SM

__host__ __device__ constexpr int act_swz(int row) {
  return (((row >> 2) & 3) << 1) ^ (row & 1) ^ ((row & 2) << 1);
}

// A warp's 8 x 4 block of threads. Lanes that differ in bit 0 share lane_x and
// lanes that differ in bit 1 share lane_y: with either, a 128-bit shared load
// takes 2 cycles of the 128-byte data path instead of the 4 of a broadcast
// between 8-lane groups (measured: x = lane & 7 and y = lane >> 3 take 4 and 2).
__device__ __forceinline__ int lane_x(int lane) { return (lane >> 1) & 7; }
__device__ __forceinline__ int lane_y(int lane) { return (lane & 1) | ((lane >> 4) << 1); }

__device__ __forceinline__ void cp16(float *dst, const float *src, int bytes = 16) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint64_t pk(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpk(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}
// two FMAs, each rounded as fmaf
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}

// acc[j][p] += w_j * (samples 2p, 2p + 1) for one k: w = 8 units, a = 8
// samples. Every other row of pairs runs backwards, so that neighbouring FMAs
// share an operand (a copy of this loop alone: 67 TFLOP/s, 65 in plain order,
// 57 with one FMA per instruction).
__device__ __forceinline__ void outer(uint64_t (&acc)[8][4], const float4 &w0, const float4 &w1,
                                      const ulonglong2 &a0, const ulonglong2 &a1) {
  const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint64_t ww = pk(w[j], w[j]);
    if (j & 1) {
      fma2(acc[j][3], ww, a1.y);
      fma2(acc[j][2], ww, a1.x);
      fma2(acc[j][1], ww, a0.y);
      fma2(acc[j][0], ww, a0.x);
    } else {
      fma2(acc[j][0], ww, a0.x);
      fma2(acc[j][1], ww, a0.y);
      fma2(acc[j][2], ww, a1.x);
      fma2(acc[j][3], ww, a1.y);
    }
  }
}

struct TrainParams {
  int64_t ns;                 // samples of this launch
  const int32_t *vox;         // [ns]
  const float4 *xyzd;         // [ns]
  int64_t n_vox, n_keys;
  float voxel_size;
  const float *centers;       // [n_vox, 3]
  const int32_t *feats;       // [n_vox, 8]
  const float4 *values;       // [n_keys, 32]
  const float *packed;        // kPacked floats
  float4 *out;                // [ns] (sigma, r, g, b)
  uint8_t *signs;             // kForwardSigns: [4][ns][16], see nsvf_field_train_forward_signs
  int32_t *err;
  // pruning (kPrune): sample s is point list[s] % bits^3 of voxel list[s] /
  // bits^3, *n_list of them (at most ns)
  const int64_t *list;
  const unsigned long long *n_list;
  int bits;
  float T, band;
  uint8_t *keep;              // [n_vox]
  int64_t *undecided;         // points within the band of T
  unsigned long long *n_undecided;
};

enum Mode { kForward, kForwardSigns, kPrune };

// offset_points' FP32 position of point i of the voxel around c (exact.cu)
__device__ __forceinline__ float point_pos(float c, int o, int bits, float hv) {
  return __fadd_rn(c, __fmul_rn(__fdiv_rn((float)(2 * o + 1 - bits), (float)(bits - 1)), hv));
}

// The weight stages, streamed in order and around.
struct Stream {
  const float *base;
  float *ws;
  int next, stage;            // next stage to issue; stage slot to read

  __device__ __forceinline__ void issue(int slot) {
    const int t = threadIdx.x;
    const float *src = base + (int64_t)next * kStage;
    cp16(ws + slot * kStage + t * 4, src + t * 4);
    cp16(ws + slot * kStage + 1024 + t * 4, src + 1024 + t * 4);
    cp_commit();
    next = next + 1 == kWStages ? 0 : next + 1;
  }
  __device__ __forceinline__ void start() {
    next = 0;
    stage = 0;
    issue(0);
    issue(1);
  }
  // The stage to read next. After the barrier every thread has left the
  // previous stage, whose slot takes the load two stages ahead. The barrier
  // also publishes what was written to shared memory before the call.
  __device__ __forceinline__ const float *take() {
    cp_wait<kStages - 2>();
    __syncthreads();
    const float *w = ws + stage * kStage;
    stage = stage + 1 == kStages ? 0 : stage + 1;
    issue(stage + 1 == kStages ? 0 : stage + 1);
    return w;
  }
};

struct Smem {
  float act[kHid * kTile];    // [unit][sample], swizzled
  float ws[kStages * kStage];
  float w4[4 * kHid];
  float bias[4 * kHid];
  float b4[4];
  float margin[kTile];        // kPrune
};

// acc = sum over k of w[k][unit] * act[k][sample], K = 16 * stages
__device__ __forceinline__ void gemm128(uint64_t (&acc)[8][4], int stages, Stream &st,
                                        const float *act, int tx, int ty) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[j][p] = 0;
#pragma unroll 1
  for (int c = 0; c < stages; ++c) {
    const float *w = st.take() + tx * 4;
    const float *a = act + c * 16 * kTile;
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const float *row = a + kk * kTile + ((ty ^ act_swz(kk)) << 2);
      const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(row);
      const ulonglong2 a1 = *reinterpret_cast<const ulonglong2 *>(row + 64);
      const float4 w0 = *reinterpret_cast<const float4 *>(w + kk * kHid);
      const float4 w1 = *reinterpret_cast<const float4 *>(w + kk * kHid + 64);
      outer(acc, w0, w1, a0, a1);
    }
  }
}

// Stores a thread's block to act (unit rows), after every thread has left it.
__device__ __forceinline__ void store_act(float *act, const float (&y)[8][8], int tx, int ty) {
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int n = (j < 4 ? 0 : 64) + tx * 4 + (j & 3);
    float *row = act + n * kTile + ((ty ^ act_swz(n)) << 2);
    *reinterpret_cast<float4 *>(row) = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
    *reinterpret_cast<float4 *>(row + 64) = make_float4(y[j][4], y[j][5], y[j][6], y[j][7]);
  }
}

template <int MODE>
__global__ void __launch_bounds__(kT, 2) field_train_kernel(const TrainParams p) {
  constexpr bool SIGNS = MODE == kForwardSigns;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem &S = *reinterpret_cast<Smem *>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int tx = (warp >> 2) * 8 + lane_x(lane), ty = (warp & 3) * 4 + lane_y(lane);
  const int unit = t & 127, half = t >> 7;
  for (int i = t; i < 4 * kHid; i += kT) {
    S.w4[i] = p.packed[kW4Off + i];
    S.bias[i] = p.packed[kBiasOff + i];
  }
  if (t < 4) S.b4[t] = p.packed[kB4Off + t];
  Stream st;
  st.base = p.packed;
  st.ws = S.ws;
  st.start();
  int64_t ns = p.ns;
  if (MODE == kPrune && (int64_t)*p.n_list < ns) ns = (int64_t)*p.n_list;
  const int64_t tiles = (ns + kTile - 1) / kTile;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t s0 = tile * kTile;
    // interpolation: 8 threads per sample, 4 channels each (interp.cu's
    // operations), into act rows 0..31
    __syncthreads();
#pragma unroll 1
    for (int it = 0; it < kTile / 32; ++it) {
      const int sl = it * 32 + (t >> 3), ch = t & 7;
      const int64_t s = s0 + sl;
      float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s < ns) {
        int64_t v;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (MODE == kPrune) {
          const int P = p.bits * p.bits * p.bits;
          v = p.list[s] / P;
          const int i = (int)(p.list[s] % P);
          if (v >= 0 && v < p.n_vox) {
            const float hv = p.voxel_size / 2.0f;
            x.x = point_pos(p.centers[v * 3 + 0], i / (p.bits * p.bits), p.bits, hv);
            x.y = point_pos(p.centers[v * 3 + 1], i / p.bits % p.bits, p.bits, hv);
            x.z = point_pos(p.centers[v * 3 + 2], i % p.bits, p.bits, hv);
          }
        } else {
          v = p.vox[s];
        }
        if (v < 0 || v >= p.n_vox) {
          if (MODE != kPrune && p.err && ch == 0) atomicOr(p.err, 4);
        } else {
          if (MODE != kPrune) x = p.xyzd[s];
          const float q[3] = {(x.x - p.centers[v * 3 + 0]) / p.voxel_size + 0.5f,
                              (x.y - p.centers[v * 3 + 1]) / p.voxel_size + 0.5f,
                              (x.z - p.centers[v * 3 + 2]) / p.voxel_size + 0.5f};
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int64_t key = p.feats[v * 8 + k];
            if (key < 0 || key >= p.n_keys) {
              if (MODE != kPrune && p.err) atomicOr(p.err, 4);
              continue;
            }
            const float w = corner_weight(q, k);
            const float4 c = __ldg(p.values + key * (kE / 4) + ch);
            e.x = fmaf(w, c.x, e.x); e.y = fmaf(w, c.y, e.y);
            e.z = fmaf(w, c.z, e.z); e.w = fmaf(w, c.w, e.w);
          }
        }
      }
      const float ev[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = ch * 4 + j;
        S.act[row * kTile + (((sl >> 2) ^ act_swz(row)) << 2) + (sl & 3)] = ev[j];
      }
    }
    uint64_t acc[8][4];
    float y[8][8];
    // hidden layers
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
      gemm128(acc, l == 0 ? kE / 16 : kHid / 16, st, S.act, tx, ty);
      uint32_t m[2] = {0, 0};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float b = S.bias[l * kHid + (j < 4 ? 0 : 64) + tx * 4 + (j & 3)];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float z0, z1;
          unpk(acc[j][q], z0, z1);
          z0 = __fadd_rn(z0, b);
          z1 = __fadd_rn(z1, b);
          if (SIGNS) {
            m[j >> 2] |= (z0 > 0.0f ? 1u : 0u) << ((j & 3) * 8 + 2 * q);
            m[j >> 2] |= (z1 > 0.0f ? 1u : 0u) << ((j & 3) * 8 + 2 * q + 1);
          }
          y[j][2 * q] = z0 <= 0.0f ? 0.0f : z0;       // NaN stays NaN
          y[j][2 * q + 1] = z1 <= 0.0f ? 0.0f : z1;
        }
      }
      if (SIGNS) {
        // units tx * 4 + 0..3 in the low half of the byte, 64 above them in
        // the high half
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int64_t q = s0 + (i < 4 ? 0 : 64) + ty * 4 + (i & 3);
          const uint32_t lo = ((m[0] >> i & 0x01010101u) * 0x01020408u) >> 24;
          const uint32_t hi = ((m[1] >> i & 0x01010101u) * 0x01020408u) >> 24;
          if (q < ns) p.signs[((int64_t)l * ns + q) * 16 + tx] = (uint8_t)(lo | hi << 4);
        }
      }
      store_act(S.act, y, tx, ty);
    }
    __syncthreads();
    if (MODE == kPrune) {
      // sigma (threads of half 0) and M = sum |W4[0]| h (half 1) of point
      // `unit`: the point is decided where sigma lies further from T than the
      // band; the others (and NaN) are listed
      float o = 0.0f;
#pragma unroll 8
      for (int k = 0; k < kHid; ++k) {
        const float a = S.act[k * kTile + (((unit >> 2) ^ act_swz(k)) << 2) + (unit & 3)];
        o = fmaf(a, half ? fabsf(S.w4[k]) : S.w4[k], o);
      }
      if (half) S.margin[unit] = o;
      __syncthreads();
      if (!half && s0 + unit < ns) {
        const float sigma = __fadd_rn(o, S.b4[0]);
        const float margin = p.band * S.margin[unit] + 1e-6f * p.T;
        const int64_t row = p.list[s0 + unit];
        if (sigma - margin > p.T)
          p.keep[row / (p.bits * p.bits * p.bits)] = 1;
        else if (!(sigma + margin < p.T))
          p.undecided[atomicAdd(p.n_undecided, 1ull)] = row;
      }
      continue;
    }
    // head: outputs 2 half, 2 half + 1 of sample `unit`
    const float *w = S.w4 + half * 2 * kHid;
    float o0 = 0.0f, o1 = 0.0f;
#pragma unroll 8
    for (int k = 0; k < kHid; ++k) {
      const float a = S.act[k * kTile + (((unit >> 2) ^ act_swz(k)) << 2) + (unit & 3)];
      o0 = fmaf(a, w[k], o0);
      o1 = fmaf(a, w[kHid + k], o1);
    }
    if (s0 + unit < ns)
      reinterpret_cast<float2 *>(p.out + s0 + unit)[half] =
          make_float2(__fadd_rn(o0, S.b4[half * 2]), __fadd_rn(o1, S.b4[half * 2 + 1]));
  }
  cp_wait<0>();
}

struct FieldWeights {
  const float *w[5], *b[5];
};

__global__ void __launch_bounds__(kT) pack_weights_kernel(FieldWeights f, float *__restrict__ out) {
  int i = blockIdx.x * kT + threadIdx.x;
  if (i >= kPacked) return;
  float v;
  constexpr int kL0 = kE * kHid, kL = kHid * kHid;
  if (i < kW4Off) {                                     // W_l transposed: [k][n]
    const int l = i < kL0 ? 0 : 1 + (i - kL0) / kL, e = i < kL0 ? i : (i - kL0) % kL;
    v = f.w[l][(e % kHid) * (l ? kHid : kE) + e / kHid];
  } else if (i < kBiasOff) {
    v = f.w[4][i - kW4Off];
  } else if (i < kB4Off) {
    v = f.b[(i - kBiasOff) / kHid][(i - kBiasOff) % kHid];
  } else {
    v = f.b[4][i - kB4Off];
  }
  out[i] = v;
}

// Valid samples (id != -1) of each row, a warp per row.
__global__ void __launch_bounds__(kT) rows_count_kernel(int64_t rays, int M,
                                                        const int32_t *__restrict__ idx,
                                                        int32_t *__restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t r = (blockIdx.x * (int64_t)kT + threadIdx.x) >> 5;
  if (r >= rays) return;
  int n = 0;
  for (int i = lane; i < M; i += 32) n += idx[r * M + i] != -1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) count[r] = n;
}

// The valid samples of each row, in slot order, to [offset[r], offset[r + 1]).
__global__ void __launch_bounds__(kT) rows_pack_kernel(
    int64_t rays, int M, const int32_t *__restrict__ idx, const float *__restrict__ xyz,
    const float *__restrict__ dists, const float *__restrict__ depths,
    const int64_t *__restrict__ offset, int32_t *__restrict__ vox, float4 *__restrict__ xyzd,
    float *__restrict__ depth) {
  const int lane = threadIdx.x & 31;
  const int64_t r = (blockIdx.x * (int64_t)kT + threadIdx.x) >> 5;
  if (r >= rays) return;
  int64_t pos = offset[r];
  for (int base = 0; base < M; base += 32) {
    const int64_t e = r * M + base + lane;
    const int32_t v = base + lane < M ? idx[e] : -1;
    const unsigned m = __ballot_sync(0xffffffffu, v != -1);
    if (v != -1) {
      const int64_t q = pos + __popc(m & ((1u << lane) - 1u));
      vox[q] = v;
      xyzd[q] = make_float4(xyz[e * 3], xyz[e * 3 + 1], xyz[e * 3 + 2], dists[e]);
      depth[q] = depths[e];
    }
    pos += __popc(m);
  }
}

// The points of `in` whose voxel is not kept yet, to `out` (any order).
__global__ void __launch_bounds__(kT) undecided_kernel(
    const int64_t *__restrict__ in, const unsigned long long *__restrict__ n_in, int64_t cap, int P,
    int64_t n_vox, const uint8_t *__restrict__ keep, int64_t *__restrict__ out,
    unsigned long long *__restrict__ n_out) {
  const int64_t n = (int64_t)*n_in < cap ? (int64_t)*n_in : cap;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * kT;
  for (int64_t base = blockIdx.x * (int64_t)kT; base < n; base += stride) {
    const int64_t i = base + threadIdx.x;
    int64_t row = 0;
    bool live = i < n;
    if (live) {
      row = in[i];
      const int64_t v = row / P;
      live = row >= 0 && v < n_vox && !keep[v];
    }
    const unsigned m = __ballot_sync(0xffffffffu, live);
    unsigned long long at = 0;
    if (m && lane == 0) at = atomicAdd(n_out, (unsigned long long)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (live) out[at + __popc(m & ((1u << lane) - 1u))] = row;
  }
}

template <int MODE>
int launch_train(const TrainParams &p, int64_t blocks, cudaStream_t s) {
  if (cudaFuncSetAttribute(field_train_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(Smem)) != cudaSuccess)
    return NSVF_ERR_CUDA;
  field_train_kernel<MODE><<<(int)blocks, kT, sizeof(Smem), s>>>(p);
  return nsvf_launch_status();
}

}  // namespace

extern "C" {

int nsvf_train_rows_count(int64_t rays, int max_steps, const int32_t *sampled_idx, int32_t *count,
                          void *stream) {
  if (rays < 0 || max_steps < 0) return NSVF_ERR_INVALID;
  if (rays == 0) return NSVF_OK;
  if ((max_steps > 0 && !sampled_idx) || !count) return NSVF_ERR_INVALID;
  rows_count_kernel<<<nsvf_grid(rays, kT / 32), kT, 0, (cudaStream_t)stream>>>(rays, max_steps,
                                                                              sampled_idx, count);
  return nsvf_launch_status();
}

int nsvf_train_rows_pack(int64_t rays, int max_steps, const int32_t *sampled_idx, const float *xyz,
                         const float *dists, const float *depths, const int64_t *offset,
                         int32_t *voxel, float *xyz_dist, float *depth, void *stream) {
  if (rays < 0 || max_steps < 0) return NSVF_ERR_INVALID;
  if (rays == 0 || max_steps == 0) return NSVF_OK;
  if (!sampled_idx || !xyz || !dists || !depths || !offset || !voxel || !xyz_dist || !depth ||
      (((uintptr_t)xyz_dist) & 15))
    return NSVF_ERR_INVALID;
  rows_pack_kernel<<<nsvf_grid(rays, kT / 32), kT, 0, (cudaStream_t)stream>>>(
      rays, max_steps, sampled_idx, xyz, dists, depths, offset, voxel, (float4 *)xyz_dist, depth);
  return nsvf_launch_status();
}

int64_t nsvf_field_train_packed_floats(void) { return kPacked; }

int nsvf_field_train_pack(const float *const weights[5], const float *const biases[5],
                          float *packed, void *stream) {
  if (!weights || !biases || !packed) return NSVF_ERR_INVALID;
  FieldWeights f;
  for (int l = 0; l < 5; ++l) {
    if (!weights[l] || !biases[l]) return NSVF_ERR_INVALID;
    f.w[l] = weights[l];
    f.b[l] = biases[l];
  }
  pack_weights_kernel<<<nsvf_grid(kPacked, kT), kT, 0, (cudaStream_t)stream>>>(f, packed);
  return nsvf_launch_status();
}

int nsvf_field_train_forward(int64_t n_samples, const int32_t *voxel, const float *xyz_dist,
                             int64_t n_voxels, int64_t n_keys, float voxel_size,
                             const float *centers, const int32_t *feats, const float *values,
                             const float *packed, float *out, int32_t *err, void *stream) {
  return nsvf_field_train_forward_signs(n_samples, voxel, xyz_dist, n_voxels, n_keys, voxel_size,
                                        centers, feats, values, packed, out, nullptr, err, stream);
}

int nsvf_field_train_forward_signs(int64_t n_samples, const int32_t *voxel, const float *xyz_dist,
                                   int64_t n_voxels, int64_t n_keys, float voxel_size,
                                   const float *centers, const int32_t *feats,
                                   const float *values, const float *packed, float *out,
                                   uint8_t *signs, int32_t *err, void *stream) {
  if (bad_scene(n_samples, voxel, xyz_dist, n_voxels, n_keys, centers, feats, values, packed))
    return NSVF_ERR_INVALID;
  if (n_samples == 0) return NSVF_OK;
  if (!out || (((uintptr_t)out) & 15)) return NSVF_ERR_INVALID;
  TrainParams p = {};
  p.ns = n_samples;
  p.vox = voxel;
  p.xyzd = (const float4 *)xyz_dist;
  p.n_vox = n_voxels;
  p.n_keys = n_keys;
  p.voxel_size = voxel_size;
  p.centers = centers;
  p.feats = feats;
  p.values = (const float4 *)values;
  p.packed = packed;
  p.out = (float4 *)out;
  p.signs = signs;
  p.err = err;
  const int64_t tiles = (n_samples + kTile - 1) / kTile, blocks = tiles < kBlocks ? tiles : kBlocks;
  return signs ? launch_train<kForwardSigns>(p, blocks, (cudaStream_t)stream)
               : launch_train<kForward>(p, blocks, (cudaStream_t)stream);
}

int nsvf_prune_fp32_dev(int64_t n_voxels, int bits, float threshold, float band, int64_t n_keys,
                        float voxel_size, const float *centers, const int32_t *feats,
                        const float *values, const float *packed, const int64_t *list,
                        const int64_t *n_list, int64_t list_cap, uint8_t *keep, int64_t *live,
                        int64_t *n_live, int64_t *undecided, int64_t *n_undecided, void *stream) {
  if (n_voxels < 0 || bits < 2 || bits > 64 || n_keys < 1 || list_cap < 0 || !(threshold > 0.0f) ||
      !(band > 0.0f))
    return NSVF_ERR_INVALID;
  if (n_voxels == 0 || list_cap == 0) return NSVF_OK;
  if (!centers || !feats || !values || !packed || !list || !n_list || !keep || !live || !n_live ||
      !undecided || !n_undecided || live == list || undecided == live ||
      ((((uintptr_t)values) | ((uintptr_t)packed)) & 15))
    return NSVF_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t need = (list_cap + kT - 1) / kT;
  undecided_kernel<<<(int)(need < 152 * 8 ? need : 152 * 8), kT, 0, s>>>(
      list, (const unsigned long long *)n_list, list_cap, bits * bits * bits, n_voxels, keep, live,
      (unsigned long long *)n_live);
  int st = nsvf_launch_status();
  if (st != NSVF_OK) return st;
  TrainParams p = {};
  p.ns = list_cap;
  p.n_vox = n_voxels;
  p.n_keys = n_keys;
  p.voxel_size = voxel_size;
  p.centers = centers;
  p.feats = feats;
  p.values = (const float4 *)values;
  p.packed = packed;
  p.list = live;
  p.n_list = (const unsigned long long *)n_live;
  p.bits = bits;
  p.T = threshold;
  p.band = band;
  p.keep = keep;
  p.undecided = undecided;
  p.n_undecided = (unsigned long long *)n_undecided;
  return launch_train<kPrune>(p, kBlocks, s);
}

}  // extern "C"
