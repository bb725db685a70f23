// Trilinear interpolation of voxel-corner embeddings and its backward
// (embedding scatter with vectorised atomics).
//
// Reference: SparseVoxelEncoder.forward (fairnr/modules/encoder.py:578-590)
// with trilinear_interp (fairnr/data/geometry.py:195-200): for a sample x in
// voxel v with centre c, p = (x - c) / voxel_size + 0.5, corner k = 4*ix +
// 2*iy + iz (offset_points order) has weight prod_d (q_kd ? p_d : 1 - p_d)
// and emb = sum_k w_k * values[feats[v, k]]. The reference materialises the
// 8 gathered rows per sample ([Ns, 8, E]) with two F.embedding calls.
//
// Two pairs of kernels. The general ones: E / 4 threads per sample, 4 channels
// each, one sample per thread. For E = 32, the embeddings' width, 8 lanes walk
// consecutive samples (trilinear_*_run_kernel): along a ray about eight in a
// row lie in the same voxel, so its corner rows stay in registers until the
// voxel changes, and so do the backward's eight corner sums, whose float4
// atomics were the bound. Measured at 1.26 M samples: see there.
#include "interp_run.cuh"

using namespace nsvf_interp;

namespace {

constexpr int kBlock = 256;

// Voxel ids outside [0, n_vox) and corner ids outside [0, n_keys) are not
// read: the sample's embedding is 0 there and bit 2 of *err is set.
template <typename IdxT, typename FeatT>
__global__ void __launch_bounds__(kBlock) trilinear_fwd_kernel(
    int64_t ns, int e4, float voxel_size, int64_t n_vox, int64_t n_keys,
    const IdxT *__restrict__ sidx, const float *__restrict__ xyz, const float *__restrict__ centers,
    const FeatT *__restrict__ feats, const float4 *__restrict__ values, float4 *__restrict__ emb,
    int32_t *__restrict__ err) {
  int64_t t = blockIdx.x * (int64_t)kBlock + threadIdx.x;
  int64_t s = t / e4;
  int ch = (int)(t - s * e4);
  if (s >= ns) return;
  int64_t v = (int64_t)sidx[s];
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (v < 0 || v >= n_vox) {
    emb[s * e4 + ch] = acc;
    if (err && ch == 0) atomicOr(err, 4);
    return;
  }
  float p[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) p[d] = (xyz[s * 3 + d] - centers[v * 3 + d]) / voxel_size + 0.5f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    int64_t key = (int64_t)feats[v * 8 + k];
    if (key < 0 || key >= n_keys) {
      if (err) atomicOr(err, 4);
      continue;
    }
    float w = corner_w(p, k);
    float4 x = __ldg(values + key * e4 + ch);
    acc.x = fmaf(w, x.x, acc.x); acc.y = fmaf(w, x.y, acc.y);
    acc.z = fmaf(w, x.z, acc.z); acc.w = fmaf(w, x.w, acc.w);
  }
  emb[s * e4 + ch] = acc;
}

// Backward: grad_values[feats[v, k]] += w_k * g (float4 atomics), and
// optionally grad_xyz = sum_k dw_k/dx . <values_k, g>.
template <typename IdxT, typename FeatT>
__global__ void __launch_bounds__(kBlock) trilinear_bwd_kernel(
    int64_t ns, int e4, float voxel_size, int64_t n_vox, int64_t n_keys,
    const IdxT *__restrict__ sidx, const float *__restrict__ xyz, const float *__restrict__ centers,
    const FeatT *__restrict__ feats, const float4 *__restrict__ values,
    const float4 *__restrict__ grad_emb, float4 *__restrict__ grad_values,
    float *__restrict__ grad_xyz) {
  int64_t t = blockIdx.x * (int64_t)kBlock + threadIdx.x;
  int64_t s = t / e4;
  int ch = (int)(t - s * e4);
  bool live = s < ns;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  int64_t v = live ? (int64_t)sidx[s] : -1;
  if (v < 0 || v >= n_vox) live = false;
  if (live) {
    float p[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d] = (xyz[s * 3 + d] - centers[v * 3 + d]) / voxel_size + 0.5f;
    float4 g = grad_emb[s * e4 + ch];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      int64_t key = (int64_t)feats[v * 8 + k];
      if (key < 0 || key >= n_keys) continue;
      float w = corner_w(p, k);
      if (grad_values) atomicAdd(grad_values + key * e4 + ch, make_float4(w * g.x, w * g.y, w * g.z, w * g.w));
      if (grad_xyz) {
        float4 x = __ldg(values + key * e4 + ch);
        float dot = x.x * g.x + x.y * g.y + x.z * g.z + x.w * g.w;
        float a = (k & 4) ? p[0] : 1.0f - p[0];
        float b = (k & 2) ? p[1] : 1.0f - p[1];
        float c = (k & 1) ? p[2] : 1.0f - p[2];
        float sa = (k & 4) ? 1.0f : -1.0f, sb = (k & 2) ? 1.0f : -1.0f, sc = (k & 1) ? 1.0f : -1.0f;
        gx += dot * sa * b * c;
        gy += dot * a * sb * c;
        gz += dot * a * b * sc;
      }
    }
  }
  if (grad_xyz) {
    // the e4 threads of a sample are consecutive lanes: reduce over them
    unsigned mask = 0xffffffffu;
    for (int o = 1; o < e4 && o < 32; o <<= 1) {
      gx += __shfl_xor_sync(mask, gx, o);
      gy += __shfl_xor_sync(mask, gy, o);
      gz += __shfl_xor_sync(mask, gz, o);
    }
    if (s < ns && ch == 0) {
      float inv = 1.0f / voxel_size;
      grad_xyz[s * 3 + 0] = gx * inv;
      grad_xyz[s * 3 + 1] = gy * inv;
      grad_xyz[s * 3 + 2] = gz * inv;
    }
  }
}

// ------------------------------------------------------ runs, E = 32 ----
//
// A group of 8 lanes takes 4 consecutive samples, a lane 4 channels of each.
// Lane c of the first four reads sample c (voxel, position, centre) and
// divides; lane c of all eight reads corner c of the samples' voxels; the rest
// comes by shuffles. Corner rows are fetched, and the backward's corner sums
// flushed, where the voxel changes. Latency-bound (four dependent trips to L2),
// so the work per thread is kept short and the blocks small: 1.26 M samples
// along rays take 80 us forward and 141 us backward (86 us for the embeddings'
// gradient alone, 90 for the positions'), where one sample per thread took 152
// and 228 (203, 170), and groups that walk 32 samples with the next batch's
// loads in flight 85 and 222. Floor 30 and 55 us: the embeddings written; read,
// and the table updated. Blocks of 256: 84 and 148 us, of 512: 88 and 164.
template <typename IdxT, typename FeatT>
__global__ void __launch_bounds__(kRunBlock) trilinear_fwd_run_kernel(
    int64_t ns, float voxel_size, int64_t n_vox, int64_t n_keys, const IdxT *__restrict__ sidx,
    const float *__restrict__ xyz, const float *__restrict__ centers,
    const FeatT *__restrict__ feats, const float4 *__restrict__ values, float4 *__restrict__ emb,
    int32_t *__restrict__ err) {
  const int64_t t = blockIdx.x * (int64_t)kRunBlock + threadIdx.x;
  const int64_t s0 = t / kLanes * kRun;
  const int ch = threadIdx.x % kLanes;
  Group<FeatT> g;
  g.template load<3>(s0, ns, voxel_size, n_vox, n_keys, sidx, xyz, centers, feats, ch, err);
  float4 x[8];
  unsigned mask = 0;
#pragma unroll
  for (int i = 0; i < kRun; ++i) {
    float p[3];
    g.coords(i, p);
    int key[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) key[k] = __shfl_sync(0xffffffffu, g.key[i], k, kLanes);
    if (g.change(i)) {
      mask = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (key[k] >= 0) {
          x[k] = __ldg(values + (int64_t)key[k] * kLanes + ch);
          mask |= 1u << k;
        }
      }
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (mask != 0xffu && !((mask >> k) & 1u)) continue;
      const float w = corner_w(p, k);
      acc.x = fmaf(w, x[k].x, acc.x); acc.y = fmaf(w, x[k].y, acc.y);
      acc.z = fmaf(w, x[k].z, acc.z); acc.w = fmaf(w, x[k].w, acc.w);
    }
    if (s0 + i < ns) emb[(s0 + i) * kLanes + ch] = acc;
  }
}

// The corners in two halves (ix = 0, then 1), so that four rows and four sums
// are live at a time. With D_k = <values_k, g>, a half adds to grad_xyz
//   x: (-1 or 1) sum_yz b_y c_z D_yz, y: a sum_z c_z (D_1z - D_0z),
//   z: a sum_y b_y (D_y1 - D_y0).
template <typename IdxT, typename FeatT, bool GV, bool GX>
__global__ void __launch_bounds__(kRunBlock, GV && GX ? 6 : 8) trilinear_bwd_run_kernel(
    int64_t ns, float voxel_size, int64_t n_vox, int64_t n_keys, const IdxT *__restrict__ sidx,
    const float *__restrict__ xyz, const float *__restrict__ centers,
    const FeatT *__restrict__ feats, const float4 *__restrict__ values,
    const float4 *__restrict__ grad_emb, float4 *__restrict__ grad_values,
    float *__restrict__ grad_xyz) {
  const unsigned full = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)kRunBlock + threadIdx.x;
  const int64_t s0 = t / kLanes * kRun;
  const int ch = threadIdx.x % kLanes;
  float4 ge[kRun];
#pragma unroll
  for (int i = 0; i < kRun; ++i)
    ge[i] = s0 + i < ns ? grad_emb[(s0 + i) * kLanes + ch] : make_float4(0.f, 0.f, 0.f, 0.f);
  Group<FeatT> g;
  g.template load<3>(s0, ns, voxel_size, n_vox, n_keys, sidx, xyz, centers, feats, ch, nullptr);
  float d[kRun][3];
#pragma unroll
  for (int i = 0; i < kRun; ++i) d[i][0] = d[i][1] = d[i][2] = 0.0f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float4 x[4], sum[4];
    int last[4] = {-1, -1, -1, -1};          // rows of the sums
    auto flush = [&]() {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (GV && last[k] >= 0) atomicAdd(grad_values + (int64_t)last[k] * kLanes + ch, sum[k]);
    };
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
      float p[3];
      g.coords(i, p);
      int key[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) key[k] = __shfl_sync(full, g.key[i], h * 4 + k, kLanes);
      if (g.change(i)) {
        if (i > 0) flush();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          last[k] = key[k];
          sum[k] = x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (GX && key[k] >= 0) x[k] = __ldg(values + (int64_t)key[k] * kLanes + ch);
        }
      }
      const float a = h ? p[0] : 1.0f - p[0];
      const float b[2] = {1.0f - p[1], p[1]}, c[2] = {1.0f - p[2], p[2]};
      const float4 gi = ge[i];
      if (GV) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float w = a * b[k >> 1] * c[k & 1];
          sum[k].x = fmaf(w, gi.x, sum[k].x); sum[k].y = fmaf(w, gi.y, sum[k].y);
          sum[k].z = fmaf(w, gi.z, sum[k].z); sum[k].w = fmaf(w, gi.w, sum[k].w);
        }
      }
      if (GX) {
        float D[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          D[k] = last[k] < 0 ? 0.0f
                             : x[k].x * gi.x + x[k].y * gi.y + x[k].z * gi.z + x[k].w * gi.w;
        const float ex = b[0] * (c[0] * D[0] + c[1] * D[1]) + b[1] * (c[0] * D[2] + c[1] * D[3]);
        d[i][0] += h ? ex : -ex;
        d[i][1] += a * (c[0] * (D[2] - D[0]) + c[1] * (D[3] - D[1]));
        d[i][2] += a * (b[0] * (D[1] - D[0]) + b[1] * (D[3] - D[2]));
      }
    }
    flush();
  }
  if (GX) {
    // over the sample's 8 lanes, the four samples folded onto the lanes: after
    // the exchange over 4 lanes a lane holds two samples, then one
    const bool up = ch & 4, mid = ch & 2;
    float e[2][3], f[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float keep = up ? d[2 + i][c] : d[i][c], give = up ? d[i][c] : d[2 + i][c];
        e[i][c] = keep + __shfl_xor_sync(full, give, 4);
      }
      const float keep = mid ? e[1][c] : e[0][c], give = mid ? e[0][c] : e[1][c];
      f[c] = keep + __shfl_xor_sync(full, give, 2);
      f[c] += __shfl_xor_sync(full, f[c], 1);
    }
    const int64_t s = s0 + (ch >> 1);
    if (!(ch & 1) && s < ns) {
      const float inv = 1.0f / voxel_size;
      grad_xyz[s * 3 + 0] = f[0] * inv;
      grad_xyz[s * 3 + 1] = f[1] * inv;
      grad_xyz[s * 3 + 2] = f[2] * inv;
    }
  }
}

struct InterpArgs {
  int64_t ns;
  int e;
  float vs;
  int64_t n_vox, n_keys;
  const void *sidx;
  const float *xyz, *centers;
  const void *feats;
  const float *values;
};

// The run kernels take E = 32 and tables whose rows 31 bits can number.
bool use_runs(const InterpArgs &a) { return a.e == 32 && a.n_keys <= 0x7fffffff; }

int run_grid(int64_t ns) { return nsvf_grid((ns + kRun - 1) / kRun * kLanes, kRunBlock); }

template <typename IdxT, typename FeatT>
int launch_fwd(const InterpArgs &a, float *emb, int32_t *err, cudaStream_t s) {
  const int e4 = a.e / 4;
  if (use_runs(a))
    trilinear_fwd_run_kernel<IdxT, FeatT><<<run_grid(a.ns), kRunBlock, 0, s>>>(
        a.ns, a.vs, a.n_vox, a.n_keys, (const IdxT *)a.sidx, a.xyz, a.centers,
        (const FeatT *)a.feats, (const float4 *)a.values, (float4 *)emb, err);
  else
    trilinear_fwd_kernel<IdxT, FeatT><<<nsvf_grid(a.ns * e4, kBlock), kBlock, 0, s>>>(
        a.ns, e4, a.vs, a.n_vox, a.n_keys, (const IdxT *)a.sidx, a.xyz, a.centers,
        (const FeatT *)a.feats, (const float4 *)a.values, (float4 *)emb, err);
  return nsvf_launch_status();
}

template <typename IdxT, typename FeatT>
int launch_bwd(const InterpArgs &a, const float *grad_emb, float *grad_values, float *grad_xyz,
               cudaStream_t s) {
  const int e4 = a.e / 4;
  if (use_runs(a)) {
    auto kernel = grad_values && grad_xyz ? trilinear_bwd_run_kernel<IdxT, FeatT, true, true>
                  : grad_values           ? trilinear_bwd_run_kernel<IdxT, FeatT, true, false>
                                          : trilinear_bwd_run_kernel<IdxT, FeatT, false, true>;
    kernel<<<run_grid(a.ns), kRunBlock, 0, s>>>(
        a.ns, a.vs, a.n_vox, a.n_keys, (const IdxT *)a.sidx, a.xyz, a.centers,
        (const FeatT *)a.feats, (const float4 *)a.values, (const float4 *)grad_emb,
        (float4 *)grad_values, grad_xyz);
  } else {
    trilinear_bwd_kernel<IdxT, FeatT><<<nsvf_grid(a.ns * e4, kBlock), kBlock, 0, s>>>(
        a.ns, e4, a.vs, a.n_vox, a.n_keys, (const IdxT *)a.sidx, a.xyz, a.centers,
        (const FeatT *)a.feats, (const float4 *)a.values, (const float4 *)grad_emb,
        (float4 *)grad_values, grad_xyz);
  }
  return nsvf_launch_status();
}

// embed_dim / 4 must be a power of two <= 32 (E in {4, 8, ..., 128}) so the
// threads of one sample are aligned lanes of one warp.
bool bad_args(int64_t ns, int e, int idx_bytes, int feat_bytes) {
  int e4 = e / 4;
  return ns < 0 || e < 4 || (e % 4) != 0 || (e4 & (e4 - 1)) != 0 || e4 > 32 ||
         (idx_bytes != 4 && idx_bytes != 8) || (feat_bytes != 4 && feat_bytes != 8);
}

}  // namespace

extern "C" {

int nsvf_trilinear_embed(int64_t n_samples, int embed_dim, float voxel_size, int64_t n_voxels,
                         int64_t n_keys, const void *sampled_idx, int idx_bytes, const float *xyz,
                         const float *centers, const void *feats, int feat_bytes,
                         const float *values, float *emb, int32_t *err, void *stream) {
  if (bad_args(n_samples, embed_dim, idx_bytes, feat_bytes)) return NSVF_ERR_INVALID;
  if (n_samples == 0) return NSVF_OK;
  if (!sampled_idx || !xyz || !centers || !feats || !values || !emb) return NSVF_ERR_INVALID;
  if ((((uintptr_t)values) | ((uintptr_t)emb)) & 15) return NSVF_ERR_INVALID;
  InterpArgs a{n_samples, embed_dim, voxel_size, n_voxels, n_keys, sampled_idx, xyz, centers,
               feats, values};
  cudaStream_t s = (cudaStream_t)stream;
  if (idx_bytes == 8 && feat_bytes == 8) return launch_fwd<int64_t, int64_t>(a, emb, err, s);
  if (idx_bytes == 8) return launch_fwd<int64_t, int32_t>(a, emb, err, s);
  if (feat_bytes == 8) return launch_fwd<int32_t, int64_t>(a, emb, err, s);
  return launch_fwd<int32_t, int32_t>(a, emb, err, s);
}

int nsvf_trilinear_embed_backward(int64_t n_samples, int embed_dim, float voxel_size,
                                  int64_t n_voxels, int64_t n_keys, const void *sampled_idx,
                                  int idx_bytes, const float *xyz, const float *centers,
                                  const void *feats, int feat_bytes, const float *values,
                                  const float *grad_emb, float *grad_values, float *grad_xyz,
                                  void *stream) {
  if (bad_args(n_samples, embed_dim, idx_bytes, feat_bytes)) return NSVF_ERR_INVALID;
  if (n_samples == 0) return NSVF_OK;
  if (!sampled_idx || !xyz || !centers || !feats || !grad_emb || (!grad_values && !grad_xyz) ||
      (grad_xyz && !values))
    return NSVF_ERR_INVALID;
  if ((((uintptr_t)grad_emb) | ((uintptr_t)grad_values) | ((uintptr_t)values)) & 15)
    return NSVF_ERR_INVALID;
  InterpArgs a{n_samples, embed_dim, voxel_size, n_voxels, n_keys, sampled_idx, xyz, centers,
               feats, values};
  cudaStream_t s = (cudaStream_t)stream;
  if (idx_bytes == 8 && feat_bytes == 8)
    return launch_bwd<int64_t, int64_t>(a, grad_emb, grad_values, grad_xyz, s);
  if (idx_bytes == 8) return launch_bwd<int64_t, int32_t>(a, grad_emb, grad_values, grad_xyz, s);
  if (feat_bytes == 8) return launch_bwd<int32_t, int64_t>(a, grad_emb, grad_values, grad_xyz, s);
  return launch_bwd<int32_t, int32_t>(a, grad_emb, grad_values, grad_xyz, s);
}

}  // extern "C"
