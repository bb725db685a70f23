// The differentiable part of a training batch on compacted samples: FP32
// interpolation + 4 x 128 field forward, and the field's and the
// interpolation's backward with the activations recomputed.
//
// Reference: SparseVoxelEncoder.forward (fairnr/modules/encoder.py:558-592),
// the field and VolumeRenderer.forward_chunk (fairnr/modules/renderer.py:
// 94-126) under autograd.
//
// Why a kernel of its own: the field's gradient is discontinuous where a
// pre-activation changes sign, so the forward has to keep FP32 and its order
// (one fused multiply-add chain over k = 0..K-1 from zero, then the bias:
// the bits of an FP32 SIMT GEMM with a bias epilogue), which leaves the
// tensor cores out. The bound is the FP32 pipe: 53,760 FMAs a sample forward,
// four times that for a training step. A chain of library GEMMs runs it at
// about 30 TFLOP/s and moves every activation through memory once per
// elementwise operation; here a tile of 128 samples goes through all layers
// in shared memory.
//
// field_train_kernel<MODE>, 256 threads, two blocks per SM (while one gathers,
// scatters or waits for weights, the other computes):
//   * activations [unit][sample] in shared memory (64 KB), each thread an 8 x
//     8 block of (unit, sample) accumulators, two samples per fma.rn.f32x2;
//   * the weights stream through three 8 KB stages by cp.async, in one
//     packed buffer that holds them in the order in which they are used
//     (forward: W_l transposed; backward: W_l as it is), so a stage is 2,048
//     consecutive floats and the next layer's weights arrive during an
//     epilogue;
//   * rows of 16-byte groups are XOR-swizzled by act_swz(row), so that the
//     epilogue's stores (8 rows, 4 apart), the GEMM's loads (one row) and the
//     per-unit sums (consecutive rows) are all free of bank conflicts.
// The backward writes the layer inputs A_l and the pre-activation gradients
// dZ_l of a chunk of samples to memory; weight_grad_kernel contracts them
// (dW_l = dZ_l^T A_l) with 128 x 128 accumulators per block over a range of
// samples. Partial sums live in per-block slots and are added in a fixed
// order, so the field's gradients are reproducible; the embeddings' are
// float4 atomics (merged over consecutive samples of one voxel).
#include "common.cuh"

namespace {

constexpr int kT = 256;
constexpr int kTile = 128;                 // samples per tile
constexpr int kHid = 128, kE = 32;
constexpr int kStages = 3;
constexpr int kStage = 2048;               // floats per weight stage
constexpr int kFwdStages = (kE + 3 * kHid) * kHid / kStage;   // 26
constexpr int kAllStages = 2 * kFwdStages;
// packed weights: the stages, then W4 [4][128], b0..b3 [4][128], b4 [4]
constexpr int kW4Off = kAllStages * kStage;
constexpr int kBiasOff = kW4Off + 4 * kHid;
constexpr int kB4Off = kBiasOff + 4 * kHid;
constexpr int kPacked = kB4Off + 4;
constexpr int kBlocks = 2 * 152;           // two per SM
// weight_grad_kernel: blocks of layers 1..3 (each) and of layer 0, whose rows
// cost about a third
constexpr int kSplit = 90, kSplit0 = kBlocks - 3 * kSplit;
constexpr int kRows = 16, kGradStages = 4;
// per half block of field_train_kernel<kBackward>: dW4 [4][128], db0..db3 [4][128]
constexpr int kSmall = 8 * kHid;

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

// w_k for corner k, multiplied in dimension order (interp.cu)
__device__ __forceinline__ float corner_weight(const float p[3], int k) {
  const float a = (k & 4) ? p[0] : 1.0f - p[0];
  const float b = (k & 2) ? p[1] : 1.0f - p[1];
  const float c = (k & 1) ? p[2] : 1.0f - p[2];
  return a * b * c;
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
  float4 *out;                // forward: [ns] (sigma, r, g, b)
  const float4 *d_out;        // backward: [ns]
  float *acts;                // backward: A0 [rows, 32], then A1, A2, A3 [rows, 128]
  float *grads;               // backward: dZ0..dZ3 [rows, 128]
  int64_t rows;               // rows of each of these arrays (>= ns, whole tiles)
  float *small;               // backward: per half block kSmall floats
  float *db4;                 // backward: per block 4 floats
  int add;                    // backward: add to the slots (0: overwrite)
  float4 *g_values;           // backward: [n_keys, 32]
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

enum Mode { kForward, kBackward, kPrune };

// offset_points' FP32 position of point i of the voxel around c (exact.cu)
__device__ __forceinline__ float point_pos(float c, int o, int bits, float hv) {
  return __fadd_rn(c, __fmul_rn(__fdiv_rn((float)(2 * o + 1 - bits), (float)(bits - 1)), hv));
}

// The weight stages, streamed in order and around.
struct Stream {
  const float *base;
  float *ws;
  int period, next, stage;    // next stage to issue; stage slot to read

  __device__ __forceinline__ void issue(int slot) {
    const int t = threadIdx.x;
    const float *src = base + (int64_t)next * kStage;
    cp16(ws + slot * kStage + t * 4, src + t * 4);
    cp16(ws + slot * kStage + 1024 + t * 4, src + 1024 + t * 4);
    cp_commit();
    next = next + 1 == period ? 0 : next + 1;
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
  float4 dout[kTile];
  uint32_t mask[4][2][kT];    // sign bits of each thread's pre-activations
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

// Stores a thread's block to rows [sample][128] of a chunk array.
__device__ __forceinline__ void store_rows(float *out, const float (&y)[8][8], int tx, int ty) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float *row = out + (int64_t)((i < 4 ? 0 : 64) + ty * 4 + (i & 3)) * kHid + tx * 4;
    *reinterpret_cast<float4 *>(row) = make_float4(y[0][i], y[1][i], y[2][i], y[3][i]);
    *reinterpret_cast<float4 *>(row + 64) = make_float4(y[4][i], y[5][i], y[6][i], y[7][i]);
  }
}

// Sum over half the tile's samples of unit row n.
__device__ __forceinline__ float row_sum(const float *act, int n, int half) {
  const int f = act_swz(n);
  float s = 0.0f;
#pragma unroll
  for (int g = 0; g < 16; ++g) {
    const float4 v =
        *reinterpret_cast<const float4 *>(act + n * kTile + (((half * 16 + g) ^ f) << 2));
    s += (v.x + v.y) + (v.z + v.w);
  }
  return s;
}

template <int MODE>
__global__ void __launch_bounds__(kT, 2) field_train_kernel(const TrainParams p) {
  constexpr bool BWD = MODE == kBackward;
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
  st.period = BWD ? kAllStages : kFwdStages;
  st.start();
  float dw4[4] = {0.f, 0.f, 0.f, 0.f}, db[4] = {0.f, 0.f, 0.f, 0.f};
  float4 db4 = make_float4(0.f, 0.f, 0.f, 0.f);
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
          if (MODE == kForward && p.err && ch == 0) atomicOr(p.err, 4);
        } else {
          if (MODE != kPrune) x = p.xyzd[s];
          const float q[3] = {(x.x - p.centers[v * 3 + 0]) / p.voxel_size + 0.5f,
                              (x.y - p.centers[v * 3 + 1]) / p.voxel_size + 0.5f,
                              (x.z - p.centers[v * 3 + 2]) / p.voxel_size + 0.5f};
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int64_t key = p.feats[v * 8 + k];
            if (key < 0 || key >= p.n_keys) {
              if (MODE == kForward && p.err) atomicOr(p.err, 4);
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
      if (BWD) reinterpret_cast<float4 *>(p.acts)[s * (kE / 4) + ch] = e;
    }
    if (BWD && t < kTile) {
      const int64_t s = s0 + t;
      const float4 d = s < ns ? p.d_out[s] : make_float4(0.f, 0.f, 0.f, 0.f);
      S.dout[t] = d;
      db4.x += d.x; db4.y += d.y; db4.z += d.z; db4.w += d.w;
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
          if (BWD) {
            m[j >> 2] |= (z0 > 0.0f ? 1u : 0u) << ((j & 3) * 8 + 2 * q);
            m[j >> 2] |= (z1 > 0.0f ? 1u : 0u) << ((j & 3) * 8 + 2 * q + 1);
          }
          y[j][2 * q] = z0 <= 0.0f ? 0.0f : z0;       // NaN stays NaN
          y[j][2 * q + 1] = z1 <= 0.0f ? 0.0f : z1;
        }
      }
      if (BWD) {
        S.mask[l][0][t] = m[0];
        S.mask[l][1][t] = m[1];
        if (l < 3)
          store_rows(p.acts + p.rows * kE + (int64_t)l * p.rows * kHid + s0 * kHid, y, tx, ty);
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
      if (half) S.dout[unit].x = o;
      __syncthreads();
      if (!half && s0 + unit < ns) {
        const float sigma = __fadd_rn(o, S.b4[0]);
        const float margin = p.band * S.dout[unit].x + 1e-6f * p.T;
        const int64_t row = p.list[s0 + unit];
        if (sigma - margin > p.T)
          p.keep[row / (p.bits * p.bits * p.bits)] = 1;
        else if (!(sigma + margin < p.T))
          p.undecided[atomicAdd(p.n_undecided, 1ull)] = row;
      }
      continue;
    }
    if (!BWD) {
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
      continue;
    }
    // dW4 += d_out^T A4: unit `unit`, half of the samples
    {
      const int f = act_swz(unit);
#pragma unroll 4
      for (int g = 0; g < 16; ++g) {
        const int gg = half * 16 + g;
        const float4 a =
            *reinterpret_cast<const float4 *>(S.act + unit * kTile + ((gg ^ f) << 2));
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 d = S.dout[gg * 4 + i];
          dw4[0] = fmaf(av[i], d.x, dw4[0]);
          dw4[1] = fmaf(av[i], d.y, dw4[1]);
          dw4[2] = fmaf(av[i], d.z, dw4[2]);
          dw4[3] = fmaf(av[i], d.w, dw4[3]);
        }
      }
    }
    // dA4 = d_out W4
    {
      const float4 *w4 = reinterpret_cast<const float4 *>(S.w4);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 d = S.dout[(i < 4 ? 0 : 64) + ty * 4 + (i & 3)];
        const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j][i] = 0.0f;
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const float4 a = w4[o * 32 + tx], b = w4[o * 32 + 16 + tx];
          y[0][i] = fmaf(dv[o], a.x, y[0][i]); y[1][i] = fmaf(dv[o], a.y, y[1][i]);
          y[2][i] = fmaf(dv[o], a.z, y[2][i]); y[3][i] = fmaf(dv[o], a.w, y[3][i]);
          y[4][i] = fmaf(dv[o], b.x, y[4][i]); y[5][i] = fmaf(dv[o], b.y, y[5][i]);
          y[6][i] = fmaf(dv[o], b.z, y[6][i]); y[7][i] = fmaf(dv[o], b.w, y[7][i]);
        }
      }
    }
    // dZ_l = dA_{l+1} (z_l > 0), then dA_l = dZ_l W_l
#pragma unroll
    for (int l = 3; l >= 0; --l) {
      if (l < 3) {
        gemm128(acc, kHid / 16, st, S.act, tx, ty);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) unpk(acc[j][q], y[j][2 * q], y[j][2 * q + 1]);
      }
      const uint32_t m0 = S.mask[l][0][t], m1 = S.mask[l][1][t];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          y[j][i] *= (((j < 4 ? m0 : m1) >> ((j & 3) * 8 + i)) & 1u) ? 1.0f : 0.0f;
      store_rows(p.grads + (int64_t)l * p.rows * kHid + s0 * kHid, y, tx, ty);
      store_act(S.act, y, tx, ty);
      __syncthreads();
      db[l] += row_sum(S.act, unit, half);
    }
    // dA0 = dZ0 W0 [128 samples x 32 channels]: 4 samples x 4 channels a thread
    {
      const int cg = lane_x(lane), sg = warp * 4 + lane_y(lane);
      float4 g[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const float *w = st.take() + cg * 4;
        const float *a = S.act + c * 64 * kTile;
#pragma unroll 16
        for (int kk = 0; kk < 64; ++kk) {
          const float4 av = *reinterpret_cast<const float4 *>(
              a + kk * kTile + ((sg ^ act_swz(kk)) << 2));
          const float4 wv = *reinterpret_cast<const float4 *>(w + kk * kE);
          const float s4[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            g[i].x = fmaf(s4[i], wv.x, g[i].x); g[i].y = fmaf(s4[i], wv.y, g[i].y);
            g[i].z = fmaf(s4[i], wv.z, g[i].z); g[i].w = fmaf(s4[i], wv.w, g[i].w);
          }
        }
      }
      // grad_values[feats[v, k]] += w_k g, summed over the thread's
      // consecutive samples of one voxel before the atomics
      int64_t prev = -1;
      float4 sum[8];
      auto flush = [&]() {
        if (prev < 0) return;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int64_t key = p.feats[prev * 8 + k];
          if (key >= 0 && key < p.n_keys) atomicAdd(p.g_values + key * (kE / 4) + cg, sum[k]);
        }
      };
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const int64_t s = s0 + sg * 4 + i;
        int64_t v = s < ns ? (int64_t)p.vox[s] : -1;
        if (v >= p.n_vox) v = -1;
        if (v < 0) continue;
        if (v != prev) {
          flush();
          prev = v;
#pragma unroll
          for (int k = 0; k < 8; ++k) sum[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float4 x = p.xyzd[s];
        const float q[3] = {(x.x - p.centers[v * 3 + 0]) / p.voxel_size + 0.5f,
                            (x.y - p.centers[v * 3 + 1]) / p.voxel_size + 0.5f,
                            (x.z - p.centers[v * 3 + 2]) / p.voxel_size + 0.5f};
        const float4 gi = i == 0 ? g[0] : i == 1 ? g[1] : i == 2 ? g[2] : g[3];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float w = corner_weight(q, k);
          sum[k].x = fmaf(w, gi.x, sum[k].x); sum[k].y = fmaf(w, gi.y, sum[k].y);
          sum[k].z = fmaf(w, gi.z, sum[k].z); sum[k].w = fmaf(w, gi.w, sum[k].w);
        }
      }
      flush();
    }
  }
  cp_wait<0>();
  if (!BWD) return;
  float *sm = p.small + (int64_t)(blockIdx.x * 2 + half) * kSmall;
#pragma unroll
  for (int o = 0; o < 4; ++o) {
    float *a = sm + o * kHid + unit, *b = sm + (4 + o) * kHid + unit;
    *a = p.add ? *a + dw4[o] : dw4[o];
    *b = p.add ? *b + db[o] : db[o];
  }
  __syncthreads();
  if (t < kTile) S.dout[t] = db4;
  __syncthreads();
  if (t < 4) {
    float s = 0.0f;
    for (int i = 0; i < kTile; ++i) s += reinterpret_cast<const float *>(S.dout + i)[t];
    float *d = p.db4 + blockIdx.x * 4 + t;
    *d = p.add ? *d + s : s;
  }
}

// dW_l = dZ_l^T A_l over a range of the chunk's samples: blocks 0..3 kSplit - 1
// are layers 1..3 (128 x 128), the rest layer 0 (128 x 32). 16 samples per
// cp.async stage, both operands [sample][unit] as they lie in memory. Adds to
// (or overwrites) the block's slot.
__global__ void __launch_bounds__(kT, 2) weight_grad_kernel(int64_t ns, int64_t rows,
                                                            const float *__restrict__ acts,
                                                            const float *__restrict__ grads,
                                                            float *__restrict__ part, int add) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float *sx = reinterpret_cast<float *>(smem_raw);           // dZ rows
  float *sy = sx + kGradStages * kRows * kHid;               // A rows
  const int t = threadIdx.x;
  const int b = blockIdx.x;
  const int l = b < 3 * kSplit ? 1 + b / kSplit : 0;
  const int j = b < 3 * kSplit ? b % kSplit : b - 3 * kSplit;
  const int splits = l ? kSplit : kSplit0;
  const int64_t per = ((ns + splits - 1) / splits + kRows - 1) / kRows * kRows;
  const int64_t r0 = j * per < ns ? j * per : ns, r1 = r0 + per < ns ? r0 + per : ns;
  const int64_t steps = (r1 - r0 + kRows - 1) / kRows;
  const float *X = grads + (int64_t)l * rows * kHid;
  const float *Y = l ? acts + rows * kE + (int64_t)(l - 1) * rows * kHid : acts;
  const int wy = l ? kHid : kE;                              // width of A rows
  auto issue = [&](int64_t step) {
    if (step < steps) {
      const int slot = (int)(step % kGradStages);
      const int64_t base = r0 + step * kRows;
      for (int q = t; q < kRows * kHid / 4; q += kT) {
        const int64_t r = base + (q >> 5);
        cp16(sx + slot * kRows * kHid + q * 4, X + (r < r1 ? r : r0) * kHid + (q & 31) * 4,
             r < r1 ? 16 : 0);
      }
      const int w4 = wy / 4;
      for (int q = t; q < kRows * w4; q += kT) {
        const int64_t r = base + q / w4;
        cp16(sy + slot * kRows * kHid + q * 4, Y + (r < r1 ? r : r0) * wy + (q % w4) * 4,
             r < r1 ? 16 : 0);
      }
    }
    cp_commit();
  };
  for (int q = 0; q < kGradStages - 1; ++q) issue(q);
  const int lane = t & 31, warp = t >> 5;
  if (l) {
    const int tx = (warp >> 2) * 8 + lane_x(lane), ty = (warp & 3) * 4 + lane_y(lane);
    uint64_t acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = 0;
#pragma unroll 1
    for (int64_t step = 0; step < steps; ++step) {
      cp_wait<kGradStages - 2>();
      __syncthreads();
      issue(step + kGradStages - 1);
      const float *x = sx + (step % kGradStages) * kRows * kHid + ty * 4;
      const float *y = sy + (step % kGradStages) * kRows * kHid + tx * 4;
#pragma unroll
      for (int s = 0; s < kRows; ++s) {
        const float4 x0 = *reinterpret_cast<const float4 *>(x + s * kHid);
        const float4 x1 = *reinterpret_cast<const float4 *>(x + s * kHid + 64);
        const ulonglong2 y0 = *reinterpret_cast<const ulonglong2 *>(y + s * kHid);
        const ulonglong2 y1 = *reinterpret_cast<const ulonglong2 *>(y + s * kHid + 64);
        outer(acc, x0, x1, y0, y1);
      }
    }
    float *P = part + (int64_t)b * kHid * kHid;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      float *row = P + ((a < 4 ? 0 : 64) + ty * 4 + (a & 3)) * kHid + tx * 4;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 v;
        unpk(acc[a][2 * h], v.x, v.y);
        unpk(acc[a][2 * h + 1], v.z, v.w);
        float4 *d = reinterpret_cast<float4 *>(row + h * 64);
        if (add) {
          const float4 o = *d;
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        *d = v;
      }
    }
  } else {
    const int kg = lane_x(lane), ng = warp * 4 + lane_y(lane);   // 4 channels, 4 units
    float4 g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int64_t step = 0; step < steps; ++step) {
      cp_wait<kGradStages - 2>();
      __syncthreads();
      issue(step + kGradStages - 1);
      const float *x = sx + (step % kGradStages) * kRows * kHid + ng * 4;
      const float *y = sy + (step % kGradStages) * kRows * kHid + kg * 4;
#pragma unroll
      for (int s = 0; s < kRows; ++s) {
        const float4 xv = *reinterpret_cast<const float4 *>(x + s * kHid);
        const float4 yv = *reinterpret_cast<const float4 *>(y + s * kE);
        const float x4[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          g[i].x = fmaf(x4[i], yv.x, g[i].x); g[i].y = fmaf(x4[i], yv.y, g[i].y);
          g[i].z = fmaf(x4[i], yv.z, g[i].z); g[i].w = fmaf(x4[i], yv.w, g[i].w);
        }
      }
    }
    float *P = part + (int64_t)3 * kSplit * kHid * kHid + (int64_t)j * kHid * kE;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 *d = reinterpret_cast<float4 *>(P + (ng * 4 + i) * kE + kg * 4);
      if (add) {
        const float4 o = *d;
        g[i].x += o.x; g[i].y += o.y; g[i].z += o.z; g[i].w += o.w;
      }
      *d = g[i];
    }
  }
  cp_wait<0>();
}

struct GradOut {
  float *w[5], *b[5];
};

// The field's gradients from the slots, each element's slots added in order.
__global__ void __launch_bounds__(kT) grad_reduce_kernel(const float *__restrict__ part,
                                                         const float *__restrict__ small,
                                                         const float *__restrict__ db4,
                                                         GradOut out) {
  int i = blockIdx.x * kT + threadIdx.x;
  const float *src;
  float *dst;
  int n, stride;
  if (i < 3 * kHid * kHid) {
    const int l = i / (kHid * kHid), e = i % (kHid * kHid);
    src = part + (int64_t)l * kSplit * kHid * kHid + e;
    n = kSplit; stride = kHid * kHid;
    dst = out.w[l + 1] + e;
  } else if ((i -= 3 * kHid * kHid) < kHid * kE) {
    src = part + (int64_t)3 * kSplit * kHid * kHid + i;
    n = kSplit0; stride = kHid * kE;
    dst = out.w[0] + i;
  } else if ((i -= kHid * kE) < kSmall) {
    src = small + i;
    n = 2 * kBlocks; stride = kSmall;
    dst = i < 4 * kHid ? out.w[4] + i : out.b[i / kHid - 4] + i % kHid;
  } else if ((i -= kSmall) < 4) {
    src = db4 + i;
    n = kBlocks; stride = 4;
    dst = out.b[4] + i;
  } else {
    return;
  }
  float s = 0.0f;
#pragma unroll 16
  for (int k = 0; k < n; ++k) s += src[(int64_t)k * stride];
  *dst = s;
}

struct FieldWeights {
  const float *w[5], *b[5];
};

__global__ void __launch_bounds__(kT) pack_weights_kernel(FieldWeights f, float *__restrict__ out) {
  int i = blockIdx.x * kT + threadIdx.x;
  if (i >= kPacked) return;
  float v;
  constexpr int kL0 = kE * kHid, kL = kHid * kHid;
  if (i < kFwdStages * kStage) {                        // W_l transposed: [k][n]
    const int l = i < kL0 ? 0 : 1 + (i - kL0) / kL, e = i < kL0 ? i : (i - kL0) % kL;
    v = f.w[l][(e % kHid) * (l ? kHid : kE) + e / kHid];
  } else if (i < kW4Off) {                              // W3, W2, W1, W0
    const int e = i - kFwdStages * kStage;
    v = e < 3 * kL ? f.w[3 - e / kL][e % kL] : f.w[0][e - 3 * kL];
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

bool bad_scene(int64_t ns, const int32_t *vox, const float *xyzd, int64_t n_vox, int64_t n_keys,
               const float *centers, const int32_t *feats, const float *values,
               const float *packed) {
  return ns < 0 || n_vox < 0 || n_keys < 0 ||
         (ns > 0 && (!vox || !xyzd || !centers || !feats || !values || !packed)) ||
         ((((uintptr_t)xyzd) | ((uintptr_t)values) | ((uintptr_t)packed)) & 15);
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

// floats of the backward's workspace besides the chunk arrays
constexpr int64_t kSlotFloats = (int64_t)3 * kSplit * kHid * kHid + (int64_t)kSplit0 * kHid * kE +
                                (int64_t)2 * kBlocks * kSmall + (int64_t)kBlocks * 4;
constexpr int64_t kRowFloats = kE + 7 * kHid;              // A0, A1..A3, dZ0..dZ3

int64_t chunk_rows(int64_t ns, int64_t chunk) {
  const int64_t c = chunk < ns ? chunk : ns;
  return (c + kTile - 1) / kTile * kTile;
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
  p.err = err;
  const int64_t tiles = (n_samples + kTile - 1) / kTile;
  return launch_train<kForward>(p, tiles < kBlocks ? tiles : kBlocks, (cudaStream_t)stream);
}

int64_t nsvf_field_train_backward_floats(int64_t n_samples, int64_t chunk_samples) {
  if (n_samples < 0 || chunk_samples < 1) return -1;
  return kSlotFloats + chunk_rows(n_samples, chunk_samples) * kRowFloats;
}

int nsvf_field_train_backward(int64_t n_samples, int64_t chunk_samples, const int32_t *voxel,
                              const float *xyz_dist, int64_t n_voxels, int64_t n_keys,
                              float voxel_size, const float *centers, const int32_t *feats,
                              const float *values, const float *packed, const float *grad_out,
                              float *workspace, int64_t workspace_floats, float *grad_values,
                              float *const grad_weights[5], float *const grad_biases[5],
                              void *stream) {
  if (bad_scene(n_samples, voxel, xyz_dist, n_voxels, n_keys, centers, feats, values, packed) ||
      chunk_samples < 1 || chunk_samples % kTile || !grad_weights || !grad_biases || !workspace ||
      (((uintptr_t)workspace) & 15))
    return NSVF_ERR_INVALID;
  if (n_samples > 0 && (!grad_out || !grad_values ||
                        ((((uintptr_t)grad_out) | ((uintptr_t)grad_values)) & 15)))
    return NSVF_ERR_INVALID;
  if (workspace_floats < nsvf_field_train_backward_floats(n_samples, chunk_samples))
    return NSVF_ERR_CAPACITY;
  GradOut g;
  for (int l = 0; l < 5; ++l) {
    if (!grad_weights[l] || !grad_biases[l]) return NSVF_ERR_INVALID;
    g.w[l] = grad_weights[l];
    g.b[l] = grad_biases[l];
  }
  cudaStream_t s = (cudaStream_t)stream;
  constexpr int smem = 2 * kGradStages * kRows * kHid * (int)sizeof(float);
  if (cudaFuncSetAttribute(weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem) != cudaSuccess)
    return NSVF_ERR_CUDA;
  const int64_t rows = chunk_rows(n_samples, chunk_samples);
  float *acts = workspace, *grads = acts + rows * (kE + 3 * kHid);
  float *part = grads + rows * 4 * kHid;
  float *small = part + (int64_t)3 * kSplit * kHid * kHid + (int64_t)kSplit0 * kHid * kE;
  float *db4 = small + (int64_t)2 * kBlocks * kSmall;
  TrainParams p = {};
  p.n_vox = n_voxels;
  p.n_keys = n_keys;
  p.voxel_size = voxel_size;
  p.centers = centers;
  p.feats = feats;
  p.values = (const float4 *)values;
  p.packed = packed;
  p.acts = acts;
  p.grads = grads;
  p.rows = rows;
  p.small = small;
  p.db4 = db4;
  p.g_values = (float4 *)grad_values;
  // (one pass without samples zeroes the slots of an empty batch)
  for (int64_t a = 0; a == 0 || a < n_samples; a += chunk_samples) {
    p.ns = n_samples - a < chunk_samples ? n_samples - a : chunk_samples;
    p.vox = voxel + a;
    p.xyzd = (const float4 *)xyz_dist + a;
    p.d_out = (const float4 *)grad_out + a;
    p.add = a > 0;
    int st = launch_train<kBackward>(p, kBlocks, s);
    if (st != NSVF_OK) return st;
    weight_grad_kernel<<<kBlocks, kT, smem, s>>>(p.ns, rows, acts, grads, part, p.add);
    st = nsvf_launch_status();
    if (st != NSVF_OK) return st;
  }
  constexpr int n_grads = 3 * kHid * kHid + kHid * kE + kSmall + 4;
  grad_reduce_kernel<<<nsvf_grid(n_grads, kT), kT, 0, s>>>(part, small, db4, g);
  return nsvf_launch_status();
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
