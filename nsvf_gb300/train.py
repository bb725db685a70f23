"""Training step of the sparse-voxel renderer (the differentiation workload):
FP32 forward and a hand-written backward with per-chunk recomputation.

The reference trains through autograd and keeps every ray chunk's graph
alive until the loss's backward (fairnr/modules/renderer.py:135-232): the
[samples, 8, 32] corner gathers and every MLP activation of the whole batch.
Here `RayBatch` is one torch.autograd.Function per batch of rays that keeps
its compacted samples (voxel ids, positions, depths, lengths: 24 bytes each),
their field values (16) and the signs of their pre-activations (64). Its
backward runs

  compositing backward     nsvf_composite_rows_backward (transmittance prefix
                           recomputed in the kernel), with the free energy's:
                           d sigma = d fe * dist * 7 where sigma > 0
  field backward           nsvf_field_train_backward: per chunk of samples,
                           interpolation and activations again, dZ = dA (Z >
                           0), dA = dZ W through all layers of a tile, then
                           dW = dZ^T A, db = sum dZ, on the tensor cores in
                           split FP32 (dW2 and dW3 in FP32 chains)
  interpolation backward   float4 atomics into the corner embeddings, from the
                           same tiles

so a batch needs one chunk's activations at a time. The field is the
workloads' 4 x 128 ReLU MLP (field.StandInField); the embeddings are the
encoder's `values` table. Fields of other widths (and tensors that are not
FP32) go through `RayChunk`, one Function per chunk of rays on cuBLAS GEMMs.

`train_step` renders a batch of rays (intersection, sampling distribution,
inverse-CDF samples: no gradient), takes the squared colour error against
the targets, backpropagates, and applies an optimizer step if one is given.
The sigma noise the reference adds in training mode
(fairnr/modules/renderer.py:119) is left out, as in evaluation mode, so that
gradients are reproducible.
"""
import ctypes

import torch
from torch.autograd import Function

from . import ext
from ._lib import LIB, check
from .functional import composite

SIGMA_SCALE = 7.0     # fairnr/modules/renderer.py:121


def _p(t):
    return t.data_ptr() if t is not None else None


def _interp(vid, xyz, centers, feats, values, voxel_size):
    ns, E = vid.numel(), values.size(-1)
    emb = torch.empty(ns, E, dtype=torch.float32, device=xyz.device)
    if ns:
        check(LIB.nsvf_trilinear_embed(
            ns, E, float(voxel_size), centers.size(0), values.size(0), _p(vid), vid.element_size(),
            _p(xyz), _p(centers), _p(feats), feats.element_size(), _p(values), _p(emb),
            _p(ext.error_word(xyz.device)), ext.ctypes_stream(xyz.device)), "trilinear_embed")
    return emb


def _mlp(emb, params):
    """Forward of the ReLU MLP; returns the output and the per-layer inputs
    A_l and pre-activations Z_l the backward needs."""
    acts, pre = [], []
    x = emb
    n = len(params) // 2
    for l in range(n):
        W, b = params[2 * l], params[2 * l + 1]
        acts.append(x)
        z = torch.addmm(b, x, W.t())
        if l < n - 1:
            pre.append(z)
            x = torch.relu(z)
        else:
            x = z
    return x, acts, pre


class RayChunk(Function):
    """(values, W0, b0, ..., W4, b4, sampled_idx [R, M], xyz [R, M, 3],
    dists [R, M], depths [R, M], centers, feats, voxel_size, kahan)
    -> (colors [R, 3], depth [R], missed [R]) of one chunk of rays."""

    @staticmethod
    def forward(ctx, values, *args):
        params = args[:10]
        sidx, xyz, dists, depths, centers, feats, voxel_size, kahan = args[10:]
        mask = sidx.ne(-1)
        vid = sidx[mask].int().contiguous()
        with torch.no_grad():
            emb = _interp(vid, xyz[mask].contiguous(), centers, feats, values, voxel_size)
            out, _, _ = _mlp(emb, params)
            fe = torch.zeros_like(dists)
            fe[mask] = torch.relu(out[:, 0]) * dists[mask] * SIGMA_SCALE
            tex = torch.zeros(dists.shape + (3,), dtype=torch.float32, device=dists.device)
            tex[mask] = out[:, 1:4]
            _, depth, missed, colors = composite(fe, tex, depths, kahan)
        ctx.save_for_backward(values, *params, sidx, xyz, dists, depths, centers, feats)
        ctx.voxel_size, ctx.kahan = float(voxel_size), bool(kahan)
        return colors, depth, missed

    @staticmethod
    def backward(ctx, g_colors, g_depth, g_missed):
        saved = ctx.saved_tensors
        values, params = saved[0], saved[1:11]
        sidx, xyz, dists, depths, centers, feats = saved[11:]
        dev = dists.device
        mask = sidx.ne(-1)
        vid = sidx[mask].int().contiguous()
        xyz_m = xyz[mask].contiguous()
        with torch.no_grad():
            # the chunk again: interpolation, activations, free energy
            emb = _interp(vid, xyz_m, centers, feats, values, ctx.voxel_size)
            out, acts, pre = _mlp(emb, params)
            sigma = out[:, 0]
            fe = torch.zeros_like(dists)
            fe[mask] = torch.relu(sigma) * dists[mask] * SIGMA_SCALE
            tex = torch.zeros(dists.shape + (3,), dtype=torch.float32, device=dev)
            tex[mask] = out[:, 1:4]
            R, M = fe.shape
            c = lambda g: g.float().contiguous() if g is not None else None
            g_fe = torch.empty_like(fe)
            g_tex = torch.empty_like(tex)
            check(LIB.nsvf_composite_backward(
                R, M, _p(fe), _p(tex), _p(depths.float().contiguous()), None, _p(c(g_depth)),
                _p(c(g_missed)), _p(c(g_colors)), _p(g_fe), _p(g_tex), int(ctx.kahan),
                ext.ctypes_stream(dev)), "composite_backward")
            d_out = torch.empty_like(out)
            d_out[:, 0] = g_fe[mask] * dists[mask] * SIGMA_SCALE * (sigma > 0)
            d_out[:, 1:4] = g_tex[mask]
            grads = [None] * 10
            dz = d_out
            n = len(params) // 2
            for l in range(n - 1, -1, -1):
                W = params[2 * l]
                grads[2 * l] = dz.t().mm(acts[l])
                grads[2 * l + 1] = dz.sum(0)
                da = dz.mm(W)
                if l > 0:
                    dz = da * (pre[l - 1] > 0)
            g_emb = da.contiguous()
            g_values = torch.zeros_like(values)
            if vid.numel():
                check(LIB.nsvf_trilinear_embed_backward(
                    vid.numel(), values.size(-1), ctx.voxel_size, centers.size(0), values.size(0),
                    _p(vid), vid.element_size(), _p(xyz_m), _p(centers), _p(feats),
                    feats.element_size(), _p(values), _p(g_emb), _p(g_values), None,
                    ext.ctypes_stream(dev)), "trilinear_embed_backward")
        return (g_values, *grads) + (None,) * 8


# Samples of two waves of nsvf_field_train_backward: 152 blocks (one per SM) of
# one 128-sample tile each. A chunk is a multiple, so that no SM idles between
# the chunks of a batch.
WAVE = 304 * 128


def chunk_samples(ns, rays, chunk_rays):
    """Samples of a backward chunk: those of chunk_rays of the batch's rays on
    average, rounded to whole waves from half a wave on and up to whole tiles of
    128 below, where the caller asks for less memory (4.4 KB a sample) than a
    wave's 170 MB at the price of idle SMs."""
    n = ns * int(chunk_rays) / max(rays, 1)
    if n >= WAVE / 2:
        return max(1, round(n / WAVE)) * WAVE
    return max(1, -(-int(n) // 128)) * 128


def _ptrs(tensors):
    return (ctypes.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])


class RayBatch(Function):
    """(values, W0, b0, ..., W4, b4, sampled_idx [R, M], xyz [R, M, 3],
    dists [R, M], depths [R, M], centers, feats, voxel_size, kahan,
    chunk_rays) -> (colors [R, 3], depth [R], missed [R]) of a batch of rays.
    chunk_samples(...) samples are recomputed at a time in the backward."""

    @staticmethod
    def forward(ctx, values, *args):
        params = args[:10]
        sidx, xyz, dists, depths, centers, feats, voxel_size, kahan, chunk_rays = args[10:]
        dev = values.device
        stream = ext.ctypes_stream(dev)
        R, M = sidx.shape
        count = torch.empty(R, dtype=torch.int32, device=dev)
        check(LIB.nsvf_train_rows_count(R, M, _p(sidx), _p(count), stream), "train_rows_count")
        offset = torch.zeros(R + 1, dtype=torch.int64, device=dev)
        torch.cumsum(count, 0, out=offset[1:])
        ns = int(offset[R])
        f = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=dev)
        vox = torch.empty(max(ns, 1), dtype=torch.int32, device=dev)
        xyzd, depth, field = f(max(ns, 1), 4), f(max(ns, 1)), f(max(ns, 1), 4)
        signs = torch.empty(4, max(ns, 1), 16, dtype=torch.uint8, device=dev) \
            if any(ctx.needs_input_grad) else None
        if ns:
            check(LIB.nsvf_train_rows_pack(R, M, _p(sidx), _p(xyz), _p(dists), _p(depths),
                                           _p(offset), _p(vox), _p(xyzd), _p(depth), stream),
                  "train_rows_pack")
            packed = RayBatch._packed(params, stream)
            check(LIB.nsvf_field_train_forward_signs(
                ns, _p(vox), _p(xyzd), centers.size(0), values.size(0), float(voxel_size),
                _p(centers), _p(feats), _p(values), _p(packed), _p(field), _p(signs),
                _p(ext.error_word(dev)), stream), "field_train_forward")
        colors, out_depth, missed = f(R, 3), f(R), f(R)
        check(LIB.nsvf_composite_rows(R, _p(offset), _p(field), _p(xyzd), _p(depth), SIGMA_SCALE,
                                      _p(colors), _p(out_depth), _p(missed), int(bool(kahan)),
                                      stream), "composite_rows")
        ctx.save_for_backward(values, *params, vox, xyzd, depth, offset, field, signs, centers,
                              feats)
        ctx.voxel_size, ctx.kahan, ctx.ns = float(voxel_size), bool(kahan), ns
        ctx.chunk = chunk_samples(ns, R, chunk_rays)
        return colors, out_depth, missed

    @staticmethod
    def _packed(params, stream):
        packed = torch.empty(int(LIB.nsvf_field_train_packed_floats()), dtype=torch.float32,
                             device=params[0].device)
        check(LIB.nsvf_field_train_pack(_ptrs(params[0::2]), _ptrs(params[1::2]), _p(packed),
                                        stream), "field_train_pack")
        return packed

    @staticmethod
    def backward(ctx, g_colors, g_depth, g_missed):
        saved = ctx.saved_tensors
        values, params = saved[0], saved[1:11]
        vox, xyzd, depth, offset, field, signs, centers, feats = saved[11:]
        dev = values.device
        stream = ext.ctypes_stream(dev)
        R, ns = offset.numel() - 1, ctx.ns
        c = lambda g: g.float().contiguous() if g is not None else None
        g_colors, g_depth, g_missed = c(g_colors), c(g_depth), c(g_missed)
        with torch.no_grad():
            g_field = torch.empty_like(field)
            check(LIB.nsvf_composite_rows_backward(
                R, _p(offset), _p(field), _p(xyzd), _p(depth), SIGMA_SCALE, _p(g_colors),
                _p(g_depth), _p(g_missed), _p(g_field), int(ctx.kahan), stream),
                "composite_rows_backward")
            g_values = torch.zeros_like(values)
            grads = [torch.empty_like(t) for t in params]
            n = int(LIB.nsvf_field_train_backward_floats(ns, ctx.chunk))
            work = torch.empty(n, dtype=torch.float32, device=dev)
            packed = RayBatch._packed(params, stream)
            check(LIB.nsvf_field_train_backward(
                ns, ctx.chunk, _p(vox), _p(xyzd), centers.size(0), values.size(0), ctx.voxel_size,
                _p(centers), _p(feats), _p(values), _p(packed), _p(signs), _p(g_field), _p(work),
                n, _p(g_values), _ptrs(grads[0::2]), _ptrs(grads[1::2]), _p(ext.error_word(dev)),
                stream),
                "field_train_backward")
        return (g_values, *grads) + (None,) * 9


FIELD_SHAPES = [(128, 32), (128,)] + [(128, 128), (128,)] * 3 + [(4, 128), (4,)]


def _batch_ok(values, params, sidx, xyz, dists, depths, centers, feats):
    """RayBatch takes FP32 tensors on one GPU, the 4 x 128 field and 32
    channels in 16-byte aligned rows; anything else goes through RayChunk."""
    if [tuple(t.shape) for t in params] != FIELD_SHAPES or values.dim() != 2 or \
            values.size(1) != 32 or sidx.dim() != 2 or xyz.shape != (*sidx.shape, 3) or \
            dists.shape != sidx.shape or depths.shape != sidx.shape or \
            centers.dim() != 2 or centers.size(1) != 3 or feats.shape != (centers.size(0), 8):
        return False
    if not all(t.is_cuda and t.dtype == torch.float32 and t.device == values.device
               for t in (values, *params, xyz, dists, depths, centers)):
        return False
    return sidx.device == feats.device == values.device and not sidx.is_floating_point() and \
        values.data_ptr() % 16 == 0 and all(t.is_contiguous() for t in (values, *params)) and \
        not torch.is_autocast_enabled()


def field_params(field):
    out = []
    for lin in field.layers:
        out += [lin.weight, lin.bias]
    return out


@torch.no_grad()
def sample_rays(encoder, ray_start, ray_dir, states=None):
    """Intersection, the sampling distribution (slot-order sums) and the
    inverse-CDF samples of a batch of rays (ray_start, ray_dir [R, 3]):
    returns (hit mask [R], sampled_idx, depths, dists [R_hit, M], xyz
    [R_hit, M, 3]). No gradient flows through the geometry."""
    if states is None:
        states = encoder.precompute(id=None)
    R = ray_dir.shape[0]
    _, _, inter, hits = encoder.ray_intersect(
        ray_start.reshape(1, 1, -1, 3).expand(1, 1, R, 3).contiguous() if ray_start.dim() == 2
        else ray_start.reshape(1, 1, 1, 3), ray_dir.reshape(1, 1, R, 3),
        {k: (v.unsqueeze(0) if v is not None else None) for k, v in states.items()})
    inter['probs'], inter['steps'] = ext.ray_probs(inter['intersected_voxel_idx'],
                                                   inter['min_depth'], inter['max_depth'],
                                                   encoder.step_size)
    hits = hits.reshape(-1)
    # the hit rays' rows, found once: indexing by the mask finds them (and
    # waits for their number) for each of seven tensors again
    rows = hits.nonzero()[:, 0]
    sub = {k: (v.reshape(-1, v.shape[-1]) if v.dim() == 3 else v.reshape(-1))[rows]
           for k, v in inter.items()}
    smp = encoder.ray_sample(sub)
    o = ray_start.reshape(-1, 3)
    o = o[rows] if o.shape[0] == R else o.expand(rows.numel(), 3)
    d = ray_dir.reshape(-1, 3)[rows]
    xyz = o[:, None, :] + d[:, None, :] * smp['sampled_point_depth'][..., None]
    return hits, smp['sampled_point_voxel_idx'], smp['sampled_point_depth'], \
        smp['sampled_point_distance'], xyz.contiguous()


def render_batch(encoder, field, ray_start, ray_dir, chunk_rays=1024, states=None, kahan=False,
                 samples=None):
    """Colours [R, 3] of a batch of rays through RayBatch or RayChunk (differentiable
    with respect to the encoder's `values` and the field's parameters), with
    the background filled in for missed rays and the missed part of hit
    rays (fairnr/models/nsvf.py:89-110)."""
    if states is None:
        states = encoder.precompute(id=None)
    if samples is None:
        samples = sample_rays(encoder, ray_start, ray_dir, states)
    hits, sidx, depths, dists, xyz = samples
    values = encoder.values.weight
    centers = states['voxel_center_xyz'].float().contiguous()
    feats = states['voxel_vertex_idx'].int().contiguous()
    params = field_params(field)
    R = ray_dir.shape[0]
    bg = field.bg_color.bg_color.float()
    colors_hit, missed_hit = [], []
    n = sidx.shape[0]
    starts = range(0, n, chunk_rays)
    if starts and _batch_ok(values, params, sidx, xyz, dists, depths, centers, feats):
        c, _, m = RayBatch.apply(values, *params, sidx.int().contiguous(), xyz.contiguous(),
                                 dists.contiguous(), depths.contiguous(), centers, feats,
                                 float(encoder.voxel_size), kahan, chunk_rays)
        colors_hit, missed_hit, starts = [c], [m], ()
    for i in starts:
        c, _, m = RayChunk.apply(values, *params, sidx[i:i + chunk_rays].contiguous(),
                                 xyz[i:i + chunk_rays].contiguous(),
                                 dists[i:i + chunk_rays].contiguous(),
                                 depths[i:i + chunk_rays].contiguous(), centers, feats,
                                 float(encoder.voxel_size), kahan)
        colors_hit.append(c)
        missed_hit.append(m)
    colors = bg.expand(R, 3).clone()
    if n:
        ch = torch.cat(colors_hit) + torch.cat(missed_hit)[:, None] * bg
        colors = colors.masked_scatter(hits[:, None].expand(R, 3), ch)
    return colors


def train_step(encoder, field, ray_start, ray_dir, target, optimizer=None, chunk_rays=1024,
               states=None, samples=None):
    """One training step: render the batch, loss = sum of squared colour
    errors against `target` [R, 3], backward (per-chunk recomputation,
    hand-written kernels), optimizer step (if given). Returns the loss."""
    if optimizer is not None:
        optimizer.zero_grad(set_to_none=True)
    colors = render_batch(encoder, field, ray_start, ray_dir, chunk_rays, states, samples=samples)
    loss = ((colors - target) ** 2).sum()
    loss.backward()
    if optimizer is not None:
        optimizer.step()
    return loss.detach()
