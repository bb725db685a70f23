// Backward of the 4 x 128 FP32 field and of the interpolation below it, on
// the tensor cores in split FP32.
//
// Reference: SparseVoxelEncoder.forward (fairnr/modules/encoder.py:558-592)
// and the field under autograd.
//
// The split. Every element of a GEMM operand is cut into three bf16 slices,
// each rounded to nearest, after its row (its K elements) was scaled by a power
// of two to |x| < 1: all 24 bits of the element, whatever else its row holds,
// down to 2^-109 of the row's largest. Of the nine products of slices the six
// of orders 0 to 2 (in steps of 2^-8) are taken; the others are 2^-23 of the
// element's product at most and 2^-26 typically. Two accumulators: one takes
// the first half of the products of order 0, the second one those of orders 2
// and 1 and then the other half. The tensor core's adder truncates, so that
// sums of half the length lose less: all products of order 0 in one accumulator
// doubled the errors below. The two are added once, where a chain of 128 FP32
// multiply-adds rounds 128 times.
//
// Why slices of the elements' own: on a grid common to the row (2^-8, 2^-17 and
// about 2^-26 of its largest element) the products of the first slices add up
// without any rounding, but an element of 1e-6 of the largest keeps few bits.
// Gradients of units that are active only in samples behind a surface were
// off by up to 2e-5 of the sum of their terms' absolute values, and everything
// by 4 % in a field whose units differ by 2^24 in size.
//
// A row with an element that is not finite (or of 2^126 and more) gets the
// scale NaN: its results are NaN and each of them is then computed by the
// FP32 chain.
//
// Errors against float64 over 128 to 200,000 samples (gradients alike,
// log-normal of sigma 6, a few 1e6 times the others, units of 2^-12 to 2^12 in
// size): 1.1e-7 to 3.2e-7 of the norm, FP32 GEMMs 1.9e-7 to 1.5e-6; single
// elements, relative to the sum of their terms' absolute values, 0.2 to 0.95 of
// the GEMMs' in the root mean square. In batches with far samples FP32 GEMMs
// over chunks leave up to 3.4e-5 of the norm; layers 2 and 3, where that is more
// than 1e-5, are summed as the GEMMs sum them (weight_chain_kernel).
//
// Measured on 1.40 M samples: 5.5 ms (the interpolation 0.3, field_bwd_kernel 2.4,
// weight_chain_kernel 1.8, weight_grad_kernel 1.0; all on the FP32 pipe took
// 6.7 + 2.7 ms, at 41 and 50 of the pipe's 66 TFLOP/s).
//
// field_bwd_kernel: a tile of 128 samples per block and one block per SM: the
// layers again (the ReLU signs are the forward's own, which are exact), then
// dZ_l = dA_{l+1} (z_l > 0), dA_l = dZ_l W_l. TMEM lane = sample, so a row's
// largest element is found by the four threads that hold it, and its slices go
// to tensor memory as the next layer's A operand, which leaves shared memory
// for the weights of two layers. The layer inputs A_l and the gradients dZ_l
// go to memory as [unit][sample] of a tile (every store a whole line), beside
// the MMAs. Bound: the chain MMA (340 of 64 cycles) -> epilogue -> slices (about
// 2k cycles each) of the one tile that fits an SM, eight times a tile, 61k
// cycles; the stores fill the MMAs' time (64 KB a layer at 27 bytes a cycle).
// A lane of the computing warps as the issuer: 0.8 ms more, behind its warp's
// share of the stores.
// weight_grad_kernel (layers 0, 1 and the head): dW_l = dZ_l^T A_l, db_l = sum
// dZ_l: K runs over the 128 samples of a tile, rows are units. FP32 accumulation
// over tiles in registers, one slot per block, the slots added in a fixed order.
// The FP32 rows of the next tile arrive by cp.async while a tile is sliced.
// Bound: the instructions and the barriers of slicing and draining, 11k cycles a
// tile of layer 1, of which the MMAs run beside 3.1k and the 128 KB from memory
// 5.6k.
#include "interp_run.cuh"
#include "tc_common.cuh"
#include "train_common.cuh"

using namespace nsvf_tc;
using namespace nsvf_train;

namespace {

constexpr int kPlane = kHid * kHid * 2;    // bytes of a slice of a 128 x 128 operand
constexpr int kSmallOp = kHid * kE * 2;    // of a 128 x 32 or 32 x 128 one
// The weight operands in the order of their use: W0..W3 (rows = units), then
// W3^T, W2^T, W1^T, W0^T (rows = inputs), three slices each.
__host__ __device__ constexpr int op_plane(int op) { return op % 7 ? kPlane : kSmallOp; }
__host__ __device__ constexpr int op_off(int op) {
  return op ? 3 * kSmallOp + (op - 1) * 3 * kPlane : 0;
}
constexpr int kSliceBytes = op_off(7) + 3 * kSmallOp;
constexpr int kScales = 7 * kHid + kE;     // a power of two per row of every operand
constexpr int kSliceFloats = kSliceBytes / 4 + kScales;

// rows of 128 samples of a tile in memory: A0 (32), A1..A4, dZ0..dZ3, dA0 as
// [sample][32], and the scales of A0's samples (row_scale)
constexpr int kDA0 = kE + 8 * kHid, kScale = kDA0 + kE, kRows = kScale + 1;
__host__ __device__ constexpr int a_row(int l) { return l ? kE + (l - 1) * kHid : 0; }
__host__ __device__ constexpr int dz_row(int l) { return kE + 4 * kHid + l * kHid; }

// weight_grad_kernel's blocks, in proportion to a tile's time: layer 1 (11k
// cycles), layer 0 (0.70 of that) and the head (0.67: an MMA of 16 columns takes
// 45 of the 64 cycles that one of 128 takes).
constexpr int kSplit1 = 64, kSplit0 = 45, kSplit4 = 43;
static_assert(kSplit1 + kSplit0 + kSplit4 == kSMs, "one block per SM");
// weight_chain_kernel's blocks of layers 2 and 3 (each), with two chains per
// element, and the longest chain (in additions) that goes on from one chunk into
// the next: that of an FP32 GEMM over a chunk of 1,024 rays is about 8,700
constexpr int kChains = kSMs / 2;
constexpr int64_t kChainLimit = 9216;

// threads of the two tensor-core kernels that compute; a fifth warpgroup's
// first lane issues the MMAs. Of the 640 x 96 registers at the launch (61,440)
// the computing warpgroups take 512 x 112 and the fifth keeps 128 x 32.
constexpr int kBT = 512, kMmaWarp = kBT / 32, kThreads = kBT + 128;
constexpr int kQ = kHid / 4;               // units of a thread's quarter of a row
constexpr uint32_t kAccCols = 128;         // columns between the two accumulators
constexpr uint32_t kACol = 256;            // field_bwd_kernel: A's slices, 64 columns each

__device__ __forceinline__ uint64_t pk(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {   // a - b
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(b), "l"(pk(-1.0f, -1.0f)), "l"(a));
  return d;
}
// two bf16 as two floats
__device__ __forceinline__ uint64_t widen(uint32_t v) {
  return pk(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// The three bf16 slices of x0, x1 scaled by inv (|x inv| < 1), each rounded to
// nearest: both differences are exact, and the three add up to x inv wherever
// that is above 2^-109.
__device__ __forceinline__ void slice2(float x0, float x1, float inv, uint32_t &h, uint32_t &m,
                                       uint32_t &l) {
  const uint64_t t = mul2(pk(x0, x1), pk(inv, inv));
  auto pack = [](uint64_t v) {
    return pack_bf16x2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
  };
  h = pack(t);
  const uint64_t r = sub2(t, widen(h));
  m = pack(r);
  l = pack(sub2(r, widen(m)));
}

__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;\n" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// The power of two above a row's largest element, whose biased exponent is e
// (NaN for a row that the slices cannot hold), and its reciprocal.
__device__ __forceinline__ uint32_t exponent(float m) { return (__float_as_uint(m) >> 23) & 255u; }
__device__ __forceinline__ float row_scale(uint32_t e) {
  return __uint_as_float(e < 253u ? (e + 1u) << 23 : 0x7fffffffu);
}
__device__ __forceinline__ float reciprocal(float scale) {
  return scale == scale ? __uint_as_float((254u << 23) - __float_as_uint(scale)) : 0.0f;
}
__device__ __forceinline__ float row_scale(uint32_t e, float &inv) {
  const float s = row_scale(e);
  inv = reciprocal(s);
  return s;
}

// Adds the products of three slices each of A (128 rows) and B, K = 16 KS, to
// the accumulators (first: to zero), those of order 0 with k < 16 KS0 to the
// first one and all others to the second; issued by one thread. A's slices are in
// tensor memory at column `a`, KS * 8 columns apart (two elements per column),
// B's in shared memory at `b`. All addresses are constants beyond these: with
// a loop of computed descriptors a MMA took 105 cycles to issue and 64 to run.
template <int KS, int B_PLANE, int N, int KS0>
__device__ __forceinline__ void issue_split_ts(uint32_t tmem, uint32_t a, uint32_t b,
                                               bool first) {
  constexpr uint32_t idesc = idesc_bf16_f32(kTile, N);
  uint64_t bd = sdesc(b, 128u, KS * 256u);
  asm volatile("" : "+l"(bd), "+r"(a));
#pragma unroll
  for (int o = 2; o >= 0; --o)
#pragma unroll
    for (int i = 0; i <= o; ++i)
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const bool low = o == 0 && k < KS0;
        mma_bf16_ts(tmem + (low ? 0u : kAccCols), a + (uint32_t)(i * KS * 8 + 8 * k),
                    bd + (uint32_t)((o - i) * B_PLANE / 16 + 16 * k), idesc,
                    first && i == 0 && k == 0 && (o == 2 || low) ? 0u : 1u);
      }
}

// A barrier of the computing threads: whether `ok` holds for all of them.
__device__ __forceinline__ bool sync_and(bool ok) { return barrier_and<kBT>(ok); }
// This warp's slices are written (every thread past its fences).
__device__ __forceinline__ void slices_ready(uint64_t *bar) {
  fence_before_sync();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// sum over k of x[k xs] w[k ws] in FP32, one fused multiply-add after the
// other: the elements that the slices cannot hold. (Inlined: around a call the
// registers of the fast path moved to the stack, 0.9 of 6.0 ms.)
__device__ __forceinline__ float chain(const float *x, int64_t xs, const float *w, int64_t ws,
                                       int K) {
  float s = 0.0f;
#pragma unroll 1
  for (int k = 0; k < K; ++k) s = fmaf(x[k * xs], w[k * ws], s);
  return s;
}

// Slices of the weight operands, a block per row.
__global__ void __launch_bounds__(kHid) slice_weights_kernel(const float *__restrict__ packed,
                                                             uint8_t *__restrict__ slices,
                                                             float *__restrict__ scales) {
  __shared__ float part[kHid / 32];
  const int op = blockIdx.x / kHid, row = blockIdx.x % kHid, k = threadIdx.x;
  const int l = op < 4 ? op : 7 - op, K = op ? kHid : kE;
  float x = 0.0f;
  if (k < K) x = packed[w_off(l) + (op < 4 ? k * kHid + row : row * kHid + k)];
  float m = fabsf(x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((k & 31) == 0) part[k >> 5] = m;
  __syncthreads();
  m = max_nan(max_nan(part[0], part[1]), max_nan(part[2], part[3]));
  float inv;
  const float s = row_scale(exponent(m), inv);
  if (k == 0) scales[blockIdx.x] = s;
  if (k >= K) return;
  uint32_t h, mi, lo;
  slice2(inv == 0.0f ? 0.0f : x, 0.0f, inv, h, mi, lo);
  uint8_t *d = slices + op_off(op) + kmajor_off(row, k & ~7, K) + (k & 7) * 2;
  *reinterpret_cast<uint16_t *>(d) = (uint16_t)h;
  *reinterpret_cast<uint16_t *>(d + op_plane(op)) = (uint16_t)mi;
  *reinterpret_cast<uint16_t *>(d + 2 * op_plane(op)) = (uint16_t)lo;
}

struct InterpParams {
  int64_t ns;                 // samples of this launch
  const int32_t *vox;         // [ns]
  const float4 *xyzd;         // [ns]
  int64_t n_vox, n_keys;
  float voxel_size;
  const float *centers;       // [n_vox, 3]
  const int32_t *feats;       // [n_vox, 8]
  const float4 *values;       // [n_keys, 32]
  float *rows;                // [tiles][kRows][128]
  float4 *g_values;           // [n_keys, 32]
};

// Interpolation of a chunk as interp.cu's run kernel does it (groups of 8
// lanes, 4 consecutive samples each), to [channel][sample] of a tile: a block
// has 64 samples and turns them in shared memory. Tiles are filled up with
// zeros. Kernels of their own, this one and the next: field_bwd_kernel's one
// block per SM has no second one to wait for memory behind (8k + 13k of a
// tile's 86k cycles were these two, and three warps for them alone could not
// keep up: 123k).
constexpr int kRunSamples = nsvf_interp::kRunBlock / nsvf_interp::kLanes * nsvf_interp::kRun;
__global__ void __launch_bounds__(nsvf_interp::kRunBlock) interp_rows_kernel(const InterpParams p) {
  using namespace nsvf_interp;
  __shared__ float out[kE][kRunSamples + 1], scale[kRunSamples];
  const int t = threadIdx.x, ch = t % kLanes, sl = t / kLanes * kRun;
  Group<int32_t> g;
  g.load<4>(blockIdx.x * (int64_t)kRunSamples + sl, p.ns, p.voxel_size, p.n_vox, p.n_keys, p.vox,
            reinterpret_cast<const float *>(p.xyzd), p.centers, p.feats, ch, nullptr);
  float4 x[8];
  unsigned mask = 0;
#pragma unroll
  for (int i = 0; i < kRun; ++i) {
    float q[3];
    g.coords(i, q);
    int key[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) key[k] = __shfl_sync(0xffffffffu, g.key[i], k, kLanes);
    if (g.change(i)) {
      mask = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (key[k] >= 0) {
          x[k] = __ldg(p.values + (int64_t)key[k] * kLanes + ch);
          mask |= 1u << k;
        }
      }
    }
    float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (mask != 0xffu && !((mask >> k) & 1u)) continue;
      const float w = corner_w(q, k);
      e.x = fmaf(w, x[k].x, e.x); e.y = fmaf(w, x[k].y, e.y);
      e.z = fmaf(w, x[k].z, e.z); e.w = fmaf(w, x[k].w, e.w);
    }
    float m = max_nan(max_nan(fabsf(e.x), fabsf(e.y)), max_nan(fabsf(e.z), fabsf(e.w)));
#pragma unroll
    for (int o = 1; o < kLanes; o <<= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    out[ch * 4][sl + i] = e.x; out[ch * 4 + 1][sl + i] = e.y;
    out[ch * 4 + 2][sl + i] = e.z; out[ch * 4 + 3][sl + i] = e.w;
    if (ch == 0) scale[sl + i] = row_scale(exponent(m));
  }
  __syncthreads();
  const int64_t s = blockIdx.x * (int64_t)kRunSamples;
  float *R = p.rows + s / kTile * kRows * kTile + s % kTile;
  if (t < kRunSamples) R[kScale * kTile + t] = scale[t];
#pragma unroll
  for (int i = t; i < kE * kRunSamples; i += kRunBlock)
    R[i / kRunSamples * kTile + i % kRunSamples] = out[i / kRunSamples][i % kRunSamples];
}

// grad_values[feats[v, k]] += w_k dA0, as interp.cu's run kernel: corner sums
// over the consecutive samples of one voxel, then float4 atomics.
__global__ void __launch_bounds__(nsvf_interp::kRunBlock, 8) interp_grad_kernel(
    const InterpParams p) {
  using namespace nsvf_interp;
  const int64_t s0 = (blockIdx.x * (int64_t)kRunBlock + threadIdx.x) / kLanes * kRun;
  const int ch = threadIdx.x % kLanes;
  const float4 *G = reinterpret_cast<const float4 *>(
      p.rows + (s0 / kTile * kRows + kDA0) * kTile + s0 % kTile * kE);
  float4 ge[kRun];
#pragma unroll
  for (int i = 0; i < kRun; ++i)
    ge[i] = s0 + i < p.ns ? G[i * kLanes + ch] : make_float4(0.f, 0.f, 0.f, 0.f);
  Group<int32_t> g;
  g.load<4>(s0, p.ns, p.voxel_size, p.n_vox, p.n_keys, p.vox,
            reinterpret_cast<const float *>(p.xyzd), p.centers, p.feats, ch, nullptr);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float4 sum[4];
    int last[4] = {-1, -1, -1, -1};          // rows of the sums
    auto flush = [&]() {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (last[k] >= 0) atomicAdd(p.g_values + (int64_t)last[k] * kLanes + ch, sum[k]);
    };
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
      float q[3];
      g.coords(i, q);
      int key[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) key[k] = __shfl_sync(0xffffffffu, g.key[i], h * 4 + k, kLanes);
      if (g.change(i)) {
        if (i > 0) flush();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          last[k] = key[k];
          sum[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float w = corner_w(q, h * 4 + k);
        sum[k].x = fmaf(w, ge[i].x, sum[k].x); sum[k].y = fmaf(w, ge[i].y, sum[k].y);
        sum[k].z = fmaf(w, ge[i].z, sum[k].z); sum[k].w = fmaf(w, ge[i].w, sum[k].w);
      }
    }
    flush();
  }
}

struct BwdParams {
  int64_t ns;                 // samples of this launch
  int64_t ns_all;             // of the batch (row length of signs)
  const float *packed;        // kPacked floats
  const uint8_t *slices;      // kSliceBytes
  const float *scales;        // kScales
  const uint4 *signs;         // [4][ns_all], from this launch's first sample
  const float4 *d_out;        // [ns]
  float *rows;                // [tiles][kRows][128]
  int32_t *err;
};

struct BwdSmem {
  uint8_t b[2][3 * kPlane];   // the slices of a layer's weights and of the next one's
  float scales[kScales];
  float bias[4 * kHid];
  // the largest exponent in each quarter of a row, of this layer and of the
  // one before: a quarter may write the next layer's while another still reads
  uint8_t top[2][4][kTile];
  uint64_t mma_done, ready, loaded[2];
  uint32_t tmem;
  int abort;
};

// Slices a thread's elements of its row to tensor memory (column `a` of its
// lane on, two elements per column).
__device__ __forceinline__ void slice_row(uint32_t a, const float (&y)[kQ], float inv) {
#pragma unroll
  for (int c = 0; c < kQ / 16; ++c) {
    uint32_t h[8], m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      slice2(y[c * 16 + 2 * i], y[c * 16 + 2 * i + 1], inv, h[i], m[i], l[i]);
    __syncwarp();
    tmem_st8(a + c * 8, h);
    tmem_st8(a + kHid / 2 + c * 8, m);
    tmem_st8(a + kHid + c * 8, l);
  }
  tmem_wait_st();
}

// v = the sums of 16 (8) columns of this thread's TMEM lane
__device__ __forceinline__ void load_sums(uint32_t tmem, float (&v)[16]) {
  float a1[16];
  __syncwarp();
  tmem_ld16(tmem, v);
  tmem_ld16(tmem + kAccCols, a1);
  tmem_wait_ld();
  // (after the wait: the loads write their registers asynchronously)
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(v[i]), "+f"(a1[i]));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] += a1[i];
}

__device__ __forceinline__ void load_sums8(uint32_t tmem, float (&v)[8]) {
  uint32_t r[2][8];
  __syncwarp();
#pragma unroll
  for (int o = 0; o < 2; ++o)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[o][0]), "=r"(r[o][1]), "=r"(r[o][2]), "=r"(r[o][3]), "=r"(r[o][4]),
                   "=r"(r[o][5]), "=r"(r[o][6]), "=r"(r[o][7])
                 : "r"(tmem + o * kAccCols)
                 : "memory");
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(r[0][i]), "+r"(r[1][i]));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[0][i]) + __uint_as_float(r[1][i]);
}

__global__ void __launch_bounds__(kThreads, 1) field_bwd_kernel(const BwdParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  BwdSmem &S = *reinterpret_cast<BwdSmem *>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int row = (warp & 3) * 32 + lane, quarter = warp >> 2, c0 = quarter * kQ;
  for (int i = t; i < 4 * kHid; i += kThreads)
    S.bias[i] = p.packed[kBiasOff + i];
  for (int i = t; i < kScales; i += kThreads) S.scales[i] = p.scales[i];
  if (t == 0) {
    mbar_init(&S.mma_done, 1);
    mbar_init(&S.ready, kBT / 32);
    mbar_init(&S.loaded[0], 1);
    mbar_init(&S.loaded[1], 1);
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  constexpr uint32_t kCols = 512;
  if (warp == 0) tmem_alloc(&S.tmem, kCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = S.tmem;
  const uint32_t tmem_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  volatile int *abort = &S.abort;
  const int64_t tiles = (p.ns + kTile - 1) / kTile;
  uint32_t ph_mma = 0;
  bool ok = true;
  if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");
    // every layer: the MMAs when its slices and its weights are there, then
    // the weights of the layer after the next
    if (t == kBT && (int64_t)blockIdx.x < tiles) {
      auto load_op = [&](int op) {
        bulk_load(S.b[op & 1], p.slices + op_off(op), 3u * op_plane(op), &S.loaded[op & 1]);
      };
      uint32_t ph_load = 0;                  // of the two buffers
      load_op(0);
      load_op(1);
      for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
#pragma unroll 1
        for (int op = 0; op < 8 && ok; ++op) {
          ok = mbar_wait(&S.ready, ph_mma, abort) &&
               mbar_wait(&S.loaded[op & 1], ph_load >> (op & 1) & 1u, abort);
          if (!ok) break;
          ph_load ^= 1u << (op & 1);
          fence_after_sync();
          const uint32_t b = smem_u32(S.b[op & 1]);
          if (op == 0)
            issue_split_ts<kE / 16, kSmallOp, kHid, 1>(tmem, tmem + kACol, b, true);
          else if (op < 7)
            issue_split_ts<kHid / 16, kPlane, kHid, 4>(tmem, tmem + kACol, b, true);
          else
            issue_split_ts<kHid / 16, kSmallOp, kE, 4>(tmem, tmem + kACol, b, true);
          mma_commit(&S.mma_done);
          ok = mbar_wait(&S.mma_done, ph_mma, abort);
          ph_mma ^= 1u;
          if (ok && (op < 6 || tile + gridDim.x < tiles)) load_op((op + 2) & 7);
        }
      if (!ok) {
        // a wait ran out: give what is in flight one more limit
        if (p.err) atomicOr(p.err, 8);
        for (int i = 0; i < 2; ++i) {
          int never = 0;
          mbar_wait(&S.loaded[i], ph_load >> i & 1u, &never);
        }
        int never = 0;
        mbar_wait(&S.mma_done, ph_mma, &never);
      }
    }
    __syncwarp();
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n");
  // Waits for a layer's MMAs.
  auto finish = [&] {
    ok = mbar_wait(&S.mma_done, ph_mma, abort) && ok;
    ph_mma ^= 1u;
    fence_after_sync();
  };
  float sa = 0.0f;                           // scale of this thread's row in A
  float y[kQ];                               // its elements: units c0 + j
  // the embeddings of this thread's sample, 8 channels, and their scale
  float e[8], es;
  auto load_e = [&](int64_t tile) {
    const float *R = p.rows + tile * kRows * kTile + row;
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = R[(quarter * 8 + j) * kTile];
    es = R[kScale * kTile];
  };
  if ((int64_t)blockIdx.x < tiles) load_e(blockIdx.x);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t s0 = tile * kTile;
    float *R = p.rows + tile * kRows * kTile;
    const bool live = s0 + row < p.ns;
    {
      sa = es;
      const float inv = reciprocal(sa);
      uint32_t a[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) slice2(e[2 * i], e[2 * i + 1], inv, a[0][i], a[1][i], a[2][i]);
      __syncwarp();
#pragma unroll
      for (int o = 0; o < 3; ++o)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(
                         tmem_row + kACol + o * (kE / 2) + quarter * 4),
                     "r"(a[o][0]), "r"(a[o][1]), "r"(a[o][2]), "r"(a[o][3]));
      tmem_wait_st();
      slices_ready(&S.ready);
    }
    // a layer's signs of this thread's units: unit j at bit 8 (j / 4 % 4) +
    // j % 4 of word j / 16
    auto signs = [&](int l, uint32_t (&m)[2]) {
      uint2 w = make_uint2(0, 0);
      if (live)
        w = reinterpret_cast<const uint2 *>(p.signs + (int64_t)l * p.ns_all + s0 + row)[quarter & 1];
      m[0] = w.x >> ((quarter >> 1) * 4);
      m[1] = w.y >> ((quarter >> 1) * 4);
    };
    auto bit = [](const uint32_t (&m)[2], int j) {
      return (m[j >> 4] >> (((j >> 2) & 3) * 8 + (j & 3))) & 1u;
    };
    auto store = [&](int first_row) {
      float *out = R + (first_row + c0) * kTile + row;
#pragma unroll
      for (int j = 0; j < kQ; ++j) out[j * kTile] = y[j];
    };
    // Ends a layer: joins the row's quarters and, where `slice`, puts its
    // slices in A. top: the largest |y|, NaN where fix(j) has to give y[j]
    // again (it reads rows of memory written before the barrier). turn: 0 and 1
    // in turn, so that the next call's barrier lies between this one's reads of
    // S.top and the next write to the same half. False: unwind.
    auto rows_done = [&](float top, int turn, bool slice, auto fix) {
      auto &tops = S.top[turn];
      tops[quarter][row] = (uint8_t)exponent(top);
      if (!sync_and(ok && top == top)) {
        if (!sync_and(ok)) return false;
        if (top != top) {
          top = 0.0f;
#pragma unroll
          for (int j = 0; j < kQ; ++j) {
            if (y[j] != y[j]) y[j] = fix(j);
            top = max_nan(top, fabsf(y[j]));
          }
          tops[quarter][row] = (uint8_t)exponent(top);
        }
        sync_and(true);
      }
      float inv;
      sa = row_scale(max(max(tops[0][row], tops[1][row]), max(tops[2][row], tops[3][row])), inv);
      if (!slice) return true;
      slice_row(tmem_row + kACol + c0 / 2, y, inv);
      slices_ready(&S.ready);
      return true;
    };
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
      uint32_t m[2];
      signs(l, m);
      if (l) store(a_row(l));
      finish();
      const float *sc = S.scales + l * kHid + c0, *bias = S.bias + l * kHid + c0;
      float top = 0.0f;
#pragma unroll
      for (int c = 0; c < kQ / 16; ++c) {
        float v[16];
        load_sums(tmem_row + c0 + c * 16, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int j = c * 16 + i;
          const float z = fmaf(v[i] * sc[j], sa, bias[j]);
          y[j] = bit(m, j) || z != z ? z : 0.0f;
          top = max_nan(top, fabsf(y[j]));
        }
      }
      if (!rows_done(top, l & 1, l < 3, [&](int j) {
            const float z = chain(R + a_row(l) * kTile + row, kTile, p.packed + w_off(l) + c0 + j,
                                  kHid, l ? kHid : kE) + bias[j];
            return bit(m, j) || z != z ? z : 0.0f;
          }))
        goto out;
    }
    store(a_row(4));
    // dA4 = d_out W4
    {
      const float4 d = live ? p.d_out[s0 + row] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 *w4 = reinterpret_cast<const float4 *>(p.packed + kW4Off + c0);
#pragma unroll
      for (int j = 0; j < kQ; j += 4) {
        const float4 a = __ldg(w4 + j / 4), b = __ldg(w4 + kHid / 4 + j / 4),
                     c = __ldg(w4 + kHid / 2 + j / 4), e4 = __ldg(w4 + 3 * kHid / 4 + j / 4);
        y[j] = fmaf(d.w, e4.x, fmaf(d.z, c.x, fmaf(d.y, b.x, d.x * a.x)));
        y[j + 1] = fmaf(d.w, e4.y, fmaf(d.z, c.y, fmaf(d.y, b.y, d.x * a.y)));
        y[j + 2] = fmaf(d.w, e4.z, fmaf(d.z, c.z, fmaf(d.y, b.z, d.x * a.z)));
        y[j + 3] = fmaf(d.w, e4.w, fmaf(d.z, c.w, fmaf(d.y, b.w, d.x * a.w)));
      }
    }
#pragma unroll 1
    for (int l = 3; l >= 0; --l) {
      uint32_t m[2];
      signs(l, m);
      float top = 0.0f;
#pragma unroll
      for (int j = 0; j < kQ; ++j) {
        y[j] *= bit(m, j) ? 1.0f : 0.0f;
        top = max_nan(top, fabsf(y[j]));
      }
      if (!rows_done(top, ~l & 1, true, [&](int j) {
            if (l == 3) return y[j];
            return chain(R + dz_row(l + 1) * kTile + row, kTile,
                         p.packed + w_off(l + 1) + (c0 + j) * kHid, 1, kHid) *
                   (bit(m, j) ? 1.0f : 0.0f);
          }))
        goto out;
      const int op = 7 - l;
      store(dz_row(l));
      if (l == 1 && tile + gridDim.x < tiles) load_e(tile + gridDim.x);
      finish();
      if (l == 0) break;
      const float *sc = S.scales + op * kHid + c0;
#pragma unroll
      for (int c = 0; c < kQ / 16; ++c) {
        float v[16];
        load_sums(tmem_row + c0 + c * 16, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) y[c * 16 + i] = v[i] * sc[c * 16 + i] * sa;
      }
    }
    // dA0: 8 channels a thread
    {
      float v[8], nan = 0.0f;               // 0 or NaN
      load_sums8(tmem_row + quarter * 8, v);
      float *g = R + kDA0 * kTile + row * kE + quarter * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = v[i] * S.scales[7 * kHid + quarter * 8 + i] * sa;
        nan = max_nan(nan, v[i]);
      }
#pragma unroll
      for (int i = 0; i < 8; i += 4)
        *reinterpret_cast<float4 *>(g + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      if (!sync_and(ok && nan == nan)) {
        if (!sync_and(ok)) goto out;
#pragma unroll 1
        for (int i = 0; i < 8 && nan != nan; ++i)
          if (g[i] != g[i])
            g[i] = chain(R + dz_row(0) * kTile + row, kTile,
                         p.packed + w_off(0) + (quarter * 8 + i) * kHid, 1, kHid);
        sync_and(true);
      }
    }
  }
out:;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem, kCols);
}

// slots of partial sums (floats): weight_grad_kernel's of layer 1, layer 0 and
// the head, weight_chain_kernel's of layers 2 and 3, and its chains
constexpr int64_t kPart0 = (int64_t)kSplit1 * kHid * kHid;
constexpr int64_t kPart4 = kPart0 + (int64_t)kSplit0 * kHid * kE;
constexpr int64_t kPart2 = kPart4 + (int64_t)kSplit4 * kHid * 4;
constexpr int64_t kPartChains = kPart2 + (int64_t)2 * kChains * kHid * kHid;
constexpr int64_t kPartFloats = kPartChains + (int64_t)2 * kChains * kHid * kHid * 2;

// The two operands of a tile in FP32, and the slices of Y for half a tile's
// samples (K = 64) in two stages; X's slices are in tensor memory.
constexpr int kHalfPlane = kHid * 64 * 2;
struct GradSmem {
  float in[2][kHid * kTile];  // X, Y: rows of 32 16-byte chunks, chunk c at c ^ (row & 7)
  uint8_t y[2][3 * kHalfPlane];
  uint8_t top[2][4][kHid];    // X, Y: the largest exponent in each quarter of a row
  float ys[2][kHid];          // Y's scales, by parity of the tile
  uint64_t done, ready[2];    // ready: of a half's slices
  uint32_t tmem;
  int abort;
};

__device__ __forceinline__ void cp_async(void *dst, const void *src, int size, bool fill) {
  if (size == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
  else                                       // 4 bytes, zero where !fill
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(fill ? 4 : 0)
                 : "memory");
}

// The MMAs of half a tile, the first ones of the first half in one accumulator
// and of the second in the other.
template <int N>
__device__ __forceinline__ void issue_half(uint32_t tmem, uint32_t x, uint32_t y, int h) {
  if (h == 0) issue_split_ts<4, kHalfPlane, N, 4>(tmem, x, y, true);
  else issue_split_ts<4, kHalfPlane, N, 0>(tmem, x, y, false);
}

// dW = X^T Y of one layer over some of the chunk's tiles, X = dZ (A4 for the
// head), Y = A (d_out). A thread slices 32 samples (a quarter of each half of
// the tile) of row t % 128 of both.
__global__ void __launch_bounds__(kThreads, 1) weight_grad_kernel(int64_t ns,
                                                             const float *__restrict__ rows,
                                                             const float *__restrict__ d_out,
                                                             float *__restrict__ part,
                                                             float *__restrict__ bias_part, int add,
                                                             int32_t *err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  GradSmem &S = *reinterpret_cast<GradSmem *>(smem_raw);
  const int t = threadIdx.x, warp = t >> 5, b = blockIdx.x;
  const int l = b < kSplit1 ? 1 : b < kSplit1 + kSplit0 ? 0 : 4;
  const int j = l == 0 ? b - kSplit1 : l == 4 ? b - kSplit1 - kSplit0 : b;
  const int splits = l == 0 ? kSplit0 : l == 4 ? kSplit4 : kSplit1;
  const int ny = l == 0 ? kE : l == 4 ? 16 : kHid;           // columns of the result
  const int yrows = l == 4 ? 4 : ny;                         // rows of Y with data
  const int64_t xrow = l == 4 ? a_row(4) : dz_row(l), yrow = l == 4 ? 0 : a_row(l);
  // TMEM lane = row of X and of the result
  const int row = t & (kHid - 1), quarter = t >> 7;
  const int ncol = ny == kHid ? 32 : ny == kE || quarter < 2 ? 8 : 0;
  const int c0 = ny == kHid ? quarter * 32 : quarter * 8;
  if (t == 0) {
    mbar_init(&S.done, 1);
    mbar_init(&S.ready[0], kBT / 32);
    mbar_init(&S.ready[1], kBT / 32);
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (l == 4)                                // rows 4..15 stay zero
    for (int i = t; i < (int)sizeof(S.y) / 16; i += kThreads)
      reinterpret_cast<uint4 *>(S.y)[i] = make_uint4(0, 0, 0, 0);
  constexpr uint32_t kCols = 512;
  if (warp == 0) tmem_alloc(&S.tmem, kCols);
  fence_async_smem();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = S.tmem;
  const uint32_t tmem_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  volatile int *abort = &S.abort;
  const int64_t tiles = (ns + kTile - 1) / kTile;
  constexpr uint32_t kXCol = 2 * kAccCols, kXHalf = 3 * 32;  // slices of a half: 32 columns each
  bool ok = true;
  if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");
    if (t == kBT) {
      int64_t n = 0;
      for (int64_t tile = j; tile < tiles && ok; tile += splits, ++n)
#pragma unroll 1
        for (int h = 0; h < 2 && ok; ++h) {
          ok = mbar_wait(&S.ready[h], (uint32_t)n & 1u, abort);
          if (!ok) break;
          fence_after_sync();
          const uint32_t x = tmem + kXCol + h * kXHalf, y = smem_u32(S.y[h]);
          if (ny == kHid) issue_half<kHid>(tmem, x, y, h);
          else if (ny == kE) issue_half<kE>(tmem, x, y, h);
          else issue_half<16>(tmem, x, y, h);
          if (h == 1) mma_commit(&S.done);
        }
      if (!ok) {
        // a wait ran out: give the MMAs in flight one more limit
        int never = 0;
        if (err) atomicOr(err, 8);
        mbar_wait(&S.done, n > 0 ? (uint32_t)(n - 1) & 1u : 0u, &never);
      }
    }
    __syncwarp();
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n");
  float acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
  float sum = 0.0f, comp = 0.0f;             // of the thread's samples of its row (db), Kahan
  float v[2][32];                            // X, Y: samples h * 64 + quarter * 16 + 0..15
  float inv[2], xs = 0.0f, xs_prev = 0.0f;
  // copies of a tile's rows to S.in
  auto fetch = [&](int64_t tile) {
    const float *R = rows + tile * kRows * kTile;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (g && l == 4) {
        // sample t / 4, output t % 4
        const int64_t s = tile * kTile + (t >> 2);
        const int u = t & 3, c = (t >> 4) ^ u;
        cp_async(S.in[1] + u * kTile + c * 4 + ((t >> 2) & 3), d_out + (s < ns ? s : 0) * 4 + u, 4,
                 s < ns);
      } else {
        const float *src = R + (g ? yrow : xrow) * kTile;
        const int n = (g ? ny : kHid) * 32;
#pragma unroll
        for (int k = 0; k < kHid * 32 / kBT; ++k) {
          const int i = t + k * kBT, r = i >> 5, c = i & 31;
          if (i < n) cp_async(S.in[g] + r * kTile + ((c ^ (r & 7)) << 2), src + i * 4, 16, true);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // the fetched tile to registers, its scales; the next one on its way
  auto take = [&](int64_t next, int buf) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    sync_and(true);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (g && row >= yrows) continue;
      const float *in = S.in[g] + row * kTile;
      float m = 0.0f, s = 0.0f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int at = (c >> 2) * 16 + quarter * 4 + (c & 3);
        const float4 a = *reinterpret_cast<const float4 *>(in + ((at ^ (row & 7)) << 2));
        if (g == (l == 4)) s += (a.x + a.y) + (a.z + a.w);   // dZ (d_out): its sum for db
        v[g][c * 4] = a.x; v[g][c * 4 + 1] = a.y; v[g][c * 4 + 2] = a.z; v[g][c * 4 + 3] = a.w;
        m = max_nan(m, max_nan(max_nan(fabsf(a.x), fabsf(a.y)), max_nan(fabsf(a.z), fabsf(a.w))));
      }
      if (g == (l == 4)) {
        const float a = s - comp, w = sum + a;
        comp = fabsf(w) <= 3.4e38f ? (w - sum) - a : 0.0f;
        sum = w;
      }
      S.top[g][quarter][row] = (uint8_t)exponent(m);
    }
    ok = sync_and(ok);
    if (next < tiles) fetch(next);
    xs_prev = xs;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (g && row >= yrows) continue;
      const float sc = row_scale(max(max(S.top[g][0][row], S.top[g][1][row]),
                                     max(S.top[g][2][row], S.top[g][3][row])),
                                 inv[g]);
      if (!g) xs = sc;
      else if (quarter == 0) S.ys[buf][row] = sc;
    }
  };
  // adds the finished result of `tile` (X's scale x) to acc
  auto drain = [&](int64_t tile, int buf, float x) {
    fence_after_sync();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c * 8 >= ncol) break;
      float d[8];
      load_sums8(tmem_row + c0 + c * 8, d);
      float nan = 0.0f;                      // 0 or NaN
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        d[i] = d[i] * S.ys[buf][c0 + c * 8 + i] * x;
        nan = max_nan(nan, d[i]);
      }
      if (nan != nan) {
        const float *X = rows + (tile * kRows + xrow + row) * kTile;
        const float *Y = l == 4 ? d_out + tile * kTile * 4 : rows + (tile * kRows + yrow) * kTile;
        const int K = ns - tile * kTile < kTile ? (int)(ns - tile * kTile) : kTile;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int n = c0 + c * 8 + i;
          if (d[i] != d[i] && n < yrows) {
            d[i] = l == 4 ? chain(X, 1, Y + n, 4, K) : chain(X, 1, Y + n * kTile, 1, K);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[c * 8 + i] += d[i];
    }
  };
  int64_t n = 0;                             // tiles begun
  if (j < tiles) fetch(j);
  for (int64_t tile = j; tile < tiles; tile += splits, ++n) {
    const int buf = (int)(n & 1);
    take(tile + splits, buf);
    if (!ok) break;
    if (n > 0) {
      ok = mbar_wait(&S.done, (uint32_t)(n - 1) & 1u, abort);
      drain(tile - splits, buf ^ 1, xs_prev);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t a[3][8];
#pragma unroll
      for (int g = 1; g >= 0; --g) {
        if (g && row >= yrows) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          slice2(v[g][h * 16 + 2 * i], v[g][h * 16 + 2 * i + 1], inv[g], a[0][i], a[1][i], a[2][i]);
        if (g) {
#pragma unroll
          for (int o = 0; o < 3; ++o) {
            uint8_t *d = S.y[h] + o * kHalfPlane + kmajor_off(row, quarter * 16, 64);
            *reinterpret_cast<uint4 *>(d) = make_uint4(a[o][0], a[o][1], a[o][2], a[o][3]);
            *reinterpret_cast<uint4 *>(d + 128) = make_uint4(a[o][4], a[o][5], a[o][6], a[o][7]);
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int o = 0; o < 3; ++o) tmem_st8(tmem_row + kXCol + h * kXHalf + o * 32 + quarter * 8, a[o]);
      tmem_wait_st();
      fence_async_smem();
      slices_ready(&S.ready[h]);
    }
  }
  if (n > 0) {                               // the same n on all threads, ok not
    ok = ok && mbar_wait(&S.done, (uint32_t)(n - 1) & 1u, abort);
    if (sync_and(ok)) drain(j + (n - 1) * splits, (int)(n - 1) & 1, xs);
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  // slots: layer 1 [128][128], layer 0 [128][32], head [128][4]
  float *P = part + (l == 0 ? kPart0 : l == 4 ? kPart4 : 0) + (int64_t)j * kHid * yrows +
             (int64_t)row * yrows + c0;
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    if (i >= ncol || c0 + i >= yrows) break;
    float4 *d = reinterpret_cast<float4 *>(P + i);
    float4 o = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    if (add) {
      const float4 w = *d;
      o.x += w.x; o.y += w.y; o.z += w.z; o.w += w.w;
    }
    *d = o;
  }
  sync_and(true);
  float *const sums = S.in[0];
  sums[quarter * kHid + row] = sum;
  sync_and(true);
  if (t < kHid) {
    const float s = (sums[t] + sums[kHid + t]) + (sums[2 * kHid + t] + sums[3 * kHid + t]);
    float *d = bias_part + (int64_t)b * kHid + t;
    *d = add ? *d + s : s;
  }
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem, kCols);
}

static_assert(sizeof(BwdSmem) <= 232448 && sizeof(GradSmem) <= 232448, "shared memory");

// dW_l = dZ_l^T A_l of layers 2 and 3 in chains of FP32 multiply-adds, and db_l.
// A block takes consecutive tiles of a chunk and goes on with the chains where
// it left them in the chunk before. Thread (tx, ty) has units tx + 16 j of dZ
// and ty + 16 i of A, and per element one chain of the even and one of the odd
// samples: two samples per fma.rn.f32x2, operands as they lie in memory.
//
// Why chains: after a far sample's product an FP32 chain loses those of 2^-24
// of it and less. In a batch with far samples FP32 GEMMs over chunks of 200k
// samples (24 chains each) lose up to 3.4e-5 of dW3's and 1.5e-5 of dW2's norm
// to that, which exact sums do not. With these chains a batch's dW3 is 3.3e-6 of
// its norm (median of 100 batches of 8,192 rays; 2.4e-5 at most) from the GEMM
// path's (RayChunk) and as far from float64 as that (1.4e-5, 40 batches); in
// one chain over all 1.7 M samples, 11,200 additions, 4.7e-6 and 1.6e-5; half
// the length 6e-6 and 1.3e-5. With exact sums 3.4e-5 apart at most in 12 batches.
// Bound: the FP32 pipe; 256 us for 194,560 samples (50 of its 66 TFLOP/s): 8 x
// 8 elements a thread and all eight chunks unrolled; 8 x 4 and twice the
// threads 283, one chunk an iteration 272, rows of elements all forwards 281.
struct ChainSmem {
  float x[3][kHid * 32], y[3][kHid * 32];  // 32 samples; 16-byte chunk c of a row at c ^ (row & 7)
};
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__global__ void __launch_bounds__(kT, 1) weight_chain_kernel(int64_t ns,
                                                              const float *__restrict__ rows,
                                                              uint64_t *__restrict__ chains,
                                                              float *__restrict__ part,
                                                              float *__restrict__ bias_part,
                                                              int begin, int end, int add,
                                                              int bias_add) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  ChainSmem &S = *reinterpret_cast<ChainSmem *>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, b = blockIdx.x;
  // (lanes that differ in bit 0 share tx: see train.cu's lane_x)
  const int tx = (warp >> 2) * 8 + ((lane >> 1) & 7);
  const int ty = (warp & 3) * 4 + ((lane & 1) | ((lane >> 4) << 1));
  const int l = 2 + b / kChains, j = b % kChains;
  const int64_t tiles = (ns + kTile - 1) / kTile, per = (tiles + kChains - 1) / kChains;
  const int64_t first = j * per, last = first + per < tiles ? first + per : tiles;
  const int stages = last > first ? (int)(last - first) * 4 : 0;
  const int xrow = dz_row(l), yrow = a_row(l);
  // stage i: a quarter of a tile, zeros behind the last sample
  auto issue = [&](int i) {
    if (i < stages) {
      const int64_t tile = first + i / 4;
      const float *R = rows + tile * kRows * kTile + (i & 3) * 32 + (t & 7) * 4;
      const int64_t left = (ns - tile * kTile - (i & 3) * 32 - (t & 7) * 4) * 4;
      const int bytes = left >= 16 ? 16 : left > 0 ? (int)left : 0;
#pragma unroll
      for (int k = 0; k < kHid * 8 / kT; ++k) {
        const int r = (t >> 3) + k * (kT / 8), at = r * 32 + (((t & 7) ^ (r & 7)) << 2);
#pragma unroll
        for (int g = 0; g < 2; ++g)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                           smem_u32((g ? S.y[i % 3] : S.x[i % 3]) + at)),
                       "l"(R + (int64_t)((g ? yrow : xrow) + r) * kTile), "r"(bytes)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  issue(0);
  issue(1);
  uint64_t acc[8][8];
  uint64_t *C = chains + (int64_t)b * kHid * kHid + t;
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[n][k] = begin ? 0 : C[(n * 8 + k) * kT];
  float sum = 0.0f, comp = 0.0f;             // db: half of row t / 2 of every stage, Kahan
#pragma unroll 1
  for (int i = 0; i < stages; ++i) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    issue(i + 2);
    const float *X = S.x[i % 3] + tx * 32, *Y = S.y[i % 3] + ty * 32;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int cx = (c ^ (tx & 7)) << 2, cy = (c ^ (ty & 7)) << 2;
      ulonglong2 x[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) x[n] = *reinterpret_cast<const ulonglong2 *>(X + n * 512 + cx);
      ulonglong2 y[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) y[k] = *reinterpret_cast<const ulonglong2 *>(Y + k * 512 + cy);
      // every other row of elements backwards: neighbouring FMAs share an operand
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int n = k & 1 ? 7 - i : i;
          fma2(acc[n][k], x[n].x, y[k].x);
        }
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int n = k & 1 ? 7 - i : i;
          fma2(acc[n][k], x[n].y, y[k].y);
        }
    }
    const float *D = S.x[i % 3] + (t >> 1) * 32;
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 a =
          *reinterpret_cast<const float4 *>(D + ((((t & 1) * 4 + q) ^ ((t >> 1) & 7)) << 2));
      s += (a.x + a.y) + (a.z + a.w);
    }
    const float a = s - comp, w = sum + a;
    comp = fabsf(w) <= 3.4e38f ? (w - sum) - a : 0.0f;
    sum = w;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  float *P = part + (int64_t)b * kHid * kHid + tx * kHid + ty;
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (!end) {
        C[(n * 8 + k) * kT] = acc[n][k];
      } else {
        float &d = P[n * 16 * kHid + k * 16];
        const float w = __uint_as_float((uint32_t)acc[n][k]) +
                        __uint_as_float((uint32_t)(acc[n][k] >> 32));
        d = add ? d + w : w;
      }
    }
  const float s = sum + __shfl_xor_sync(0xffffffffu, sum, 1);
  float *d = bias_part + (int64_t)b * kHid + (t >> 1);
  if (!(t & 1)) *d = bias_add ? *d + s : s;
}

struct GradOut {
  float *w[5], *b[5];
};

// The field's gradients from the slots, each element's slots added in order.
// NaN, and NaN in grad_values, where a wait ran out (bit 3 of *err): an update
// with what was summed so far would not be noticed.
__global__ void __launch_bounds__(kT) grad_reduce_kernel(const float *__restrict__ part,
                                                         const float *__restrict__ bias_part,
                                                         GradOut out, float *__restrict__ g_values,
                                                         int64_t n_values,
                                                         const int32_t *__restrict__ err) {
  int i = blockIdx.x * kT + threadIdx.x;
  const bool failed = err && (*err & 8) != 0;
  const float nan = __int_as_float(0x7fffffff);
  if (failed)
    for (int64_t k = i; k < n_values; k += (int64_t)gridDim.x * kT) g_values[k] = nan;
  const float *src;
  float *dst;
  int n, stride;
  if (i < 3 * kHid * kHid) {
    const int l = i / (kHid * kHid) + 1, e = i % (kHid * kHid);
    src = part + (l > 1 ? kPart2 + (int64_t)(l - 2) * kChains * kHid * kHid : 0) + e;
    n = l > 1 ? kChains : kSplit1; stride = kHid * kHid;
    dst = out.w[l] + e;
  } else if ((i -= 3 * kHid * kHid) < kHid * kE) {
    src = part + kPart0 + i;
    n = kSplit0; stride = kHid * kE;
    dst = out.w[0] + i;
  } else if ((i -= kHid * kE) < kHid * 4) {
    src = part + kPart4 + i;
    n = kSplit4; stride = kHid * 4;
    dst = out.w[4] + (i & 3) * kHid + (i >> 2);
  } else if ((i -= kHid * 4) < 4 * kHid) {
    const int l = i / kHid;
    src = bias_part + (int64_t)(l == 0 ? kSplit1 : l == 1 ? 0 : kSMs + (l - 2) * kChains) * kHid +
          i % kHid;
    n = l == 0 ? kSplit0 : l == 1 ? kSplit1 : kChains; stride = kHid;
    dst = out.b[l] + i % kHid;
  } else if ((i -= 4 * kHid) < 4) {
    src = bias_part + (int64_t)(kSplit1 + kSplit0) * kHid + i;
    n = kSplit4; stride = kHid;
    dst = out.b[4] + i;
  } else {
    return;
  }
  float s = 0.0f, c = 0.0f;                  // compensated (Kahan)
#pragma unroll 8
  for (int k = 0; k < n; ++k) {
    const float a = src[(int64_t)k * stride] - c, b = s + a;
    c = fabsf(b) <= 3.4e38f ? (b - s) - a : 0.0f;
    s = b;
  }
  *dst = failed ? nan : s;
}

// floats of the workspace besides a chunk's rows
constexpr int64_t kFixedFloats = kPartFloats + (int64_t)(kSMs + 2 * kChains) * kHid + (kSliceFloats + 31) / 32 * 32;

int64_t chunk_rows(int64_t ns, int64_t chunk) {
  const int64_t c = chunk < ns ? chunk : ns;
  return (c + kTile - 1) / kTile * kTile;
}

}  // namespace

extern "C" {

int64_t nsvf_field_train_backward_floats(int64_t n_samples, int64_t chunk_samples) {
  if (n_samples < 0 || chunk_samples < 1) return -1;
  return kFixedFloats + chunk_rows(n_samples, chunk_samples) * kRows;
}

// A chunk adds as many additions to a chain as half of a block's tiles have
// samples. As many chunks go on with it as its limit allows.
int64_t nsvf_field_train_chain_chunks(int64_t n_samples, int64_t chunk_samples) {
  if (n_samples < 0 || chunk_samples < 1) return -1;
  const int64_t chunks = (n_samples + chunk_samples - 1) / chunk_samples;
  const int64_t tiles = (chunk_samples + kTile - 1) / kTile;
  const int64_t most = kChainLimit / ((tiles + kChains - 1) / kChains * (kTile / 2));
  return most < 2 || chunks < 2 ? 1 : most < chunks ? most : chunks;
}

int nsvf_field_train_backward(int64_t n_samples, int64_t chunk_samples, const int32_t *voxel,
                              const float *xyz_dist, int64_t n_voxels, int64_t n_keys,
                              float voxel_size, const float *centers, const int32_t *feats,
                              const float *values, const float *packed, const uint8_t *signs,
                              const float *grad_out, float *workspace, int64_t workspace_floats,
                              float *grad_values, float *const grad_weights[5],
                              float *const grad_biases[5], int32_t *err, void *stream) {
  if (bad_scene(n_samples, voxel, xyz_dist, n_voxels, n_keys, centers, feats, values, packed) ||
      chunk_samples < 1 || chunk_samples % kTile || !grad_weights || !grad_biases || !workspace ||
      !packed || (((uintptr_t)workspace) & 15))
    return NSVF_ERR_INVALID;
  if (n_samples > 0 &&
      (!grad_out || !grad_values || !signs ||
       ((((uintptr_t)grad_out) | ((uintptr_t)grad_values) | ((uintptr_t)signs)) & 15)))
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
  if (cudaFuncSetAttribute(field_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(BwdSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(GradSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(weight_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(ChainSmem)) != cudaSuccess)
    return NSVF_ERR_CUDA;
  float *rows = workspace;
  uint8_t *slices =
      (uint8_t *)(rows + chunk_rows(n_samples, chunk_samples) * kRows);
  float *scales = (float *)(slices + kSliceBytes);
  float *part = (float *)slices + (kSliceFloats + 31) / 32 * 32;
  float *bias_part = part + kPartFloats;
  int st;
  if (n_samples > 0) {
    slice_weights_kernel<<<kScales, kHid, 0, s>>>(packed, slices, scales);
    if ((st = nsvf_launch_status()) != NSVF_OK) return st;
  }
  BwdParams p = {};
  p.ns_all = n_samples;
  p.packed = packed;
  p.slices = slices;
  p.scales = scales;
  p.rows = rows;
  p.err = err;
  InterpParams q = {};
  q.n_vox = n_voxels;
  q.n_keys = n_keys;
  q.voxel_size = voxel_size;
  q.centers = centers;
  q.feats = feats;
  q.values = (const float4 *)values;
  q.rows = rows;
  q.g_values = (float4 *)grad_values;
  const int64_t chunks = (n_samples + chunk_samples - 1) / chunk_samples;
  const int64_t group = nsvf_field_train_chain_chunks(n_samples, chunk_samples);
  int64_t k = 0;                             // chunk
  // (one pass without samples zeroes the slots of an empty batch)
  for (int64_t a = 0; a == 0 || a < n_samples; a += chunk_samples, ++k) {
    p.ns = n_samples - a < chunk_samples ? n_samples - a : chunk_samples;
    q.ns = p.ns;
    q.vox = voxel + a;
    q.xyzd = (const float4 *)xyz_dist + a;
    p.signs = (const uint4 *)signs + a;
    p.d_out = (const float4 *)grad_out + a;
    if (p.ns > 0) {
      const int64_t tiles = (p.ns + kTile - 1) / kTile;
      interp_rows_kernel<<<nsvf_grid(tiles * kTile, kRunSamples), nsvf_interp::kRunBlock, 0, s>>>(
          q);
      if ((st = nsvf_launch_status()) != NSVF_OK) return st;
      field_bwd_kernel<<<(int)(tiles < kSMs ? tiles : kSMs), kThreads, sizeof(BwdSmem), s>>>(p);
      if ((st = nsvf_launch_status()) != NSVF_OK) return st;
      interp_grad_kernel<<<nsvf_grid(p.ns, kRunSamples), nsvf_interp::kRunBlock, 0, s>>>(q);
      if ((st = nsvf_launch_status()) != NSVF_OK) return st;
    }
    weight_grad_kernel<<<kSMs, kThreads, sizeof(GradSmem), s>>>(p.ns, rows, (const float *)p.d_out, part,
                                                          bias_part, a > 0, err);
    if ((st = nsvf_launch_status()) != NSVF_OK) return st;
    weight_chain_kernel<<<2 * kChains, kT, sizeof(ChainSmem), s>>>(
        p.ns, rows, (uint64_t *)(part + kPartChains), part + kPart2,
        bias_part + (int64_t)kSMs * kHid, k % group == 0, k % group == group - 1 || k + 1 >= chunks,
        k >= group, a > 0);
    if ((st = nsvf_launch_status()) != NSVF_OK) return st;
  }
  constexpr int n_grads = 3 * kHid * kHid + kHid * kE + 8 * kHid + 4;
  grad_reduce_kernel<<<nsvf_grid(n_grads, kT), kT, 0, s>>>(
      part, bias_part, g, grad_values, n_samples > 0 ? n_keys * kE : 0, err);
  return nsvf_launch_status();
}

}  // extern "C"
