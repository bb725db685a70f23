"""The training batch's kernels (nsvf_gb300/csrc/train.cu) at sizes around
their tiles: the FP32 field forward against a chain of cuBLAS FP32 layers
(bit for bit) and the whole batch's colours and gradients against float64
torch autograd."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene(cuda, n_vox, seed):
    g = torch.Generator().manual_seed(seed)
    vs = 0.25
    centers = torch.rand(n_vox, 3, generator=g) * 2 - 1
    feats = torch.randint(0, 3 * n_vox, (n_vox, 8), generator=g, dtype=torch.int32)
    values = torch.randn(3 * n_vox, 32, generator=g) * 0.3
    dims = [32, 128, 128, 128, 128, 4]
    params = []
    for a, b in zip(dims[:-1], dims[1:]):
        params += [torch.randn(b, a, generator=g) * a ** -0.5, torch.randn(b, generator=g) * 0.1]
    return vs, centers.to(cuda), feats.to(cuda), values.to(cuda), [p.to(cuda) for p in params]


def _rows(cuda, rays, steps, n_vox, vs, centers, seed):
    """sampled_idx with -1 both inside and at the end of the rows (and empty
    rows), positions inside the sampled voxels, increasing depths."""
    g = torch.Generator().manual_seed(seed + 1)
    idx = torch.randint(0, n_vox, (rays, steps), generator=g, dtype=torch.int32)
    runs = torch.randint(0, n_vox, (rays, max(1, steps // 5 + 1)), generator=g, dtype=torch.int32)
    idx = torch.where(torch.rand(rays, 1, generator=g) < 0.7,
                      runs.repeat_interleave(5, 1)[:, :steps], idx)
    idx[torch.rand(rays, steps, generator=g) < 0.1] = -1
    idx[torch.arange(steps)[None] >= torch.randint(0, steps + 1, (rays, 1), generator=g)] = -1
    off = (torch.rand(rays, steps, 3, generator=g) - 0.5) * vs
    idx, off = idx.to(cuda), off.to(cuda)
    xyz = centers[idx.clamp(min=0).long()] + off
    dists = torch.rand(rays, steps, generator=g).to(cuda) * 0.1
    depths = torch.rand(rays, steps, generator=g).cumsum(1).to(cuda)
    return idx, xyz.contiguous(), dists, depths


def _field64(idx, xyz, centers, feats, values, params, vs):
    m = idx.ne(-1)
    v = idx[m].long()
    p = (xyz[m] - centers[v]) / vs + 0.5
    x = 0
    for k in range(8):
        w = 1
        for d, bit in enumerate((4, 2, 1)):
            w = w * (p[:, d] if k & bit else 1 - p[:, d])
        x = x + w[:, None] * values[feats[v, k].long()]
    for l in range(5):
        x = x @ params[2 * l].t() + params[2 * l + 1]
        x = torch.relu(x) if l < 4 else x
    return m, x


# samples: below one tile, across a tile's edge, more tiles than blocks (304
# tiles of 128), and a backward in several chunks
@pytest.mark.parametrize("rays,steps,chunk_rays", [(1, 1, 1), (3, 47, 2), (130, 3, 1024),
                                                   (257, 64, 64), (900, 100, 300)])
def test_batch_matches_float64_autograd(cuda, rays, steps, chunk_rays):
    from nsvf_gb300 import ext, train
    n_vox = 97
    vs, centers, feats, values, params = _scene(cuda, n_vox, rays)
    idx, xyz, dists, depths = _rows(cuda, rays, steps, n_vox, vs, centers, rays)
    values.requires_grad_(True)
    for p in params:
        p.requires_grad_(True)
    g = torch.Generator().manual_seed(5)
    gc, gd, gm = (torch.randn(*s, generator=g).to(cuda) for s in ((rays, 3), (rays,), (rays,)))
    out = train.RayBatch.apply(values, *params, idx, xyz, dists, depths, centers, feats, vs, False,
                               chunk_rays)
    grads = torch.autograd.grad(out, [values, *params], (gc, gd, gm))
    ext.check_errors(cuda)
    v64 = values.detach().double().requires_grad_(True)
    p64 = [p.detach().double().requires_grad_(True) for p in params]
    vs32 = float(np.float32(vs))
    m, x = _field64(idx, xyz.double(), centers.double(), feats, v64, p64, vs32)
    z = torch.zeros(rays, steps, dtype=torch.float64, device=cuda)
    fe = z.masked_scatter(m, torch.relu(x[:, 0]) * dists.double()[m] * 7.0)
    tex = torch.stack([z.masked_scatter(m, x[:, 1 + c]) for c in range(3)], -1)
    T = torch.exp(-torch.cat([z[:, :1], fe[:, :-1]], 1).cumsum(1))
    pr = (1 - torch.exp(-fe)) * T
    ref = ((pr[..., None] * tex).sum(1), (pr * depths.double()).sum(1), 1 - pr.sum(1))
    ref_g = torch.autograd.grad(ref, [v64, *p64], (gc.double(), gd.double(), gm.double()))
    # FP32 sums of at most 100 terms of order 1 along a ray (colours), then of
    # all samples (gradients); a sign of a pre-activation within FP32 rounding
    # of zero (about one in 1e7 of the 512 per sample) changes a gradient by
    # one sample's share
    for a, b in zip(out, ref):
        a, b = a.detach().double(), b.detach()
        assert float((a - b).abs().max()) <= 2e-5 * (1 + float(b.abs().max()))
    for a, b in zip(grads, ref_g):
        scale = float(b.norm()) + 1e-12
        assert float((a.detach().double() - b.detach()).norm()) <= 2e-3 * scale


@pytest.mark.parametrize("ns", [100, 128, 129, 40000])
def test_forward_bits_of_a_gemm_chain(cuda, ns):
    """out = the bits of nsvf_trilinear_embed followed by torch.addmm / relu
    (FP32 cuBLAS: one fused multiply-add chain over k, then the bias), so a
    training run keeps every ReLU's sign."""
    from nsvf_gb300 import ext, train
    from nsvf_gb300._lib import LIB, check
    from nsvf_gb300.functional import trilinear_embed
    n_vox = 61
    vs, centers, feats, values, params = _scene(cuda, n_vox, ns)
    g = torch.Generator().manual_seed(ns)
    vid = torch.randint(0, n_vox, (ns,), generator=g, dtype=torch.int32).to(cuda)
    xyz = centers[vid.long()] + (torch.rand(ns, 3, generator=g).to(cuda) - 0.5) * vs
    xyzd = torch.cat([xyz, torch.ones(ns, 1, device=cuda)], 1).contiguous()
    stream = ext.ctypes_stream(cuda)
    packed = train.RayBatch._packed(params, stream)
    out = torch.empty(ns, 4, device=cuda)
    check(LIB.nsvf_field_train_forward(
        ns, vid.data_ptr(), xyzd.data_ptr(), n_vox, values.size(0), vs, centers.data_ptr(),
        feats.data_ptr(), values.data_ptr(), packed.data_ptr(), out.data_ptr(),
        ext.error_word(cuda).data_ptr(), stream), "field_train_forward")
    x = trilinear_embed(vid, xyz.contiguous(), centers, feats, values, vs)
    for l in range(5):
        x = torch.addmm(params[2 * l + 1], x, params[2 * l].t())
        x = torch.relu(x) if l < 4 else x
    ext.check_errors(cuda)
    assert torch.equal(out, x)


def _field_grads(cuda, ns, dout, seed, chunk, far=None, rescale=None):
    """The field's forward with signs and its backward on random samples, and
    the FP32 layers of the same samples: (grads, grad_values), (acts, pre,
    params, scene)."""
    from nsvf_gb300 import ext, train
    from nsvf_gb300._lib import LIB, check
    from nsvf_gb300.functional import trilinear_embed
    n_vox = 61
    vs, centers, feats, values, params = _scene(cuda, n_vox, seed)
    if rescale is not None:
        rescale(params)
    g = torch.Generator().manual_seed(seed)
    vid = torch.randint(0, n_vox, (ns,), generator=g, dtype=torch.int32).to(cuda)
    xyz = (centers[vid.long()] + (torch.rand(ns, 3, generator=g).to(cuda) - 0.5) * vs).contiguous()
    if far is not None:
        xyz[far] += 40 * vs
    xyzd = torch.cat([xyz, torch.ones(ns, 1, device=cuda)], 1).contiguous()
    stream, err = ext.ctypes_stream(cuda), ext.error_word(cuda)
    packed = train.RayBatch._packed(params, stream)
    out = torch.empty(ns, 4, device=cuda)
    signs = torch.zeros(4, ns, 16, dtype=torch.uint8, device=cuda)
    scene = (n_vox, values.size(0), vs, centers.data_ptr(), feats.data_ptr(), values.data_ptr(),
             packed.data_ptr())
    check(LIB.nsvf_field_train_forward_signs(ns, vid.data_ptr(), xyzd.data_ptr(), *scene,
                                             out.data_ptr(), signs.data_ptr(), err.data_ptr(),
                                             stream), "forward")
    n = int(LIB.nsvf_field_train_backward_floats(ns, chunk))
    work = torch.empty(n, device=cuda)
    gv, grads = torch.zeros_like(values), [torch.empty_like(p) for p in params]
    check(LIB.nsvf_field_train_backward(
        ns, chunk, vid.data_ptr(), xyzd.data_ptr(), *scene, signs.data_ptr(), dout.data_ptr(),
        work.data_ptr(), n, gv.data_ptr(), train._ptrs(grads[0::2]), train._ptrs(grads[1::2]),
        err.data_ptr(), stream), "backward")
    ext.check_errors(cuda)
    acts, pre = [trilinear_embed(vid, xyz, centers, feats, values, vs)], []
    for l in range(4):
        pre.append(torch.addmm(params[2 * l + 1], acts[-1], params[2 * l].t()))
        acts.append(torch.relu(pre[-1]))
    return (grads, gv), (acts, pre, params, (vid, xyz, centers, feats, values, vs))


def _chain_grads(acts, pre, params, dout):
    grads, dz = [None] * 10, dout
    for l in range(4, -1, -1):
        grads[2 * l], grads[2 * l + 1] = dz.t() @ acts[l], dz.sum(0)
        da = dz @ params[2 * l]
        if l:
            dz = da * (pre[l - 1] > 0)
    return grads, da


# one sample, a tile's edges, fewer tiles than splits, several chunks; the
# samples' gradients of one size, and over many orders of magnitude; samples far
# outside their voxel, whose activations are some thousand times the others',
# without a gradient of their own
@pytest.mark.parametrize("ns,spread,far", [(1, 0.0, None), (127, 4.0, None), (128, 0.0, None),
                                           (129, 1.0, None), (5000, 12.0, None),
                                           (60000, 0.0, None), (60000, 3.0, None),
                                           (128, 0.0, 17), (5000, 0.0, 100)])
def test_split_backward_against_float64(cuda, ns, spread, far):
    """The tensor-core backward against float64 with the FP32 forward's ReLU
    signs. Each of at most nine contractions in a row is good to about 2^-23
    of its result's norm, the FP32 sums over tiles and slots to a few more:
    2^-18 in all; the embeddings' float4 atomics add up to 1,000 samples."""
    g = torch.Generator().manual_seed(ns)
    dout = (torch.randn(ns, 4, generator=g) *
            torch.exp(spread * torch.randn(ns, 1, generator=g))).to(cuda)
    far = slice(far, None, far) if far else None
    if far:
        dout[far] = 0
    (grads, gv), (acts, pre, params, scene) = _field_grads(cuda, ns, dout, ns, 304 * 128, far)
    vid, xyz, centers, feats, values, vs = scene
    p64 = [p.double() for p in params]
    q = (xyz.double() - centers[vid.long()].double()) / float(np.float32(vs)) + 0.5
    w = [1, 1, 1, 1, 1, 1, 1, 1]
    for k in range(8):
        for d, bit in enumerate((4, 2, 1)):
            w[k] = w[k] * (q[:, d] if k & bit else 1 - q[:, d])
    keys = feats[vid.long()].long()
    a64 = [sum(w[k][:, None] * values.double()[keys[:, k]] for k in range(8))]
    for l in range(4):
        a64.append((a64[-1] @ p64[2 * l].t() + p64[2 * l + 1]) * (pre[l] > 0))
    ref, da = _chain_grads(a64, pre, p64, dout.double())
    ref_v = torch.zeros_like(values, dtype=torch.float64)
    for k in range(8):
        ref_v.index_add_(0, keys[:, k], w[k][:, None] * da)
    for a, b in zip([*grads, gv], [*ref, ref_v]):
        assert float((a.double() - b).norm()) <= 2.0 ** -18 * float(b.norm())


@pytest.mark.parametrize("ns,chunks", [(300, 1), (100000, 3), (2150000, 13)])
def test_weight_chains_across_chunks(cuda, ns, chunks):
    """Weight gradients of one chunk, of several that share their FP32 chains,
    and of more samples than one set of chains takes. At most 9,300 additions
    round in a chain, as a random walk by 2^-24 each: 2^-17 of the norm."""
    g = torch.Generator().manual_seed(ns)
    dout = torch.randn(ns, 4, generator=g).to(cuda)
    chunk = -(-ns // chunks) // 128 * 128 + 128
    (grads, _), (acts, pre, params, _) = _field_grads(cuda, ns, dout, ns, chunk)
    p64 = [p.double() for p in params]
    ref = [0] * 10
    for i in range(0, ns, 250000):
        s = slice(i, i + 250000)
        part, _ = _chain_grads([a[s].double() for a in acts], [z[s] for z in pre], p64,
                               dout[s].double())
        ref = [r + q for r, q in zip(ref, part)]
    for a, b in zip(grads, ref):
        assert float((a.double() - b).norm()) <= 2.0 ** -17 * float(b.norm())


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 9e37, 1e-40])
def test_split_backward_rows_the_slices_cannot_hold(cuda, value):
    """A gradient that is not finite, near the largest float, or denormal: the
    same infinities and NaNs as FP32 GEMMs, and the same finite values."""
    ns = 300
    g = torch.Generator().manual_seed(3)
    dout = torch.randn(ns, 4, generator=g)
    dout[::97, 1] = value
    dout = dout.to(cuda)
    (grads, gv), (acts, pre, params, _) = _field_grads(cuda, ns, dout, 9, 304 * 128)
    ref, _ = _chain_grads(acts, pre, params, dout)
    for a, b in zip(grads, ref):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.isinf(), b.isinf())
        m = b.isfinite()
        assert torch.equal(a[b.isinf()], b[b.isinf()])
        if m.any():
            assert float((a[m] - b[m]).double().norm()) <= 1e-5 * float(b[m].double().norm())
    if value != value or abs(value) == float("inf"):
        assert not gv.isfinite().all()


def test_other_widths_keep_the_general_path(cuda):
    """A field that is not 4 x 128 trains through RayChunk."""
    from nsvf_gb300 import train
    vs, centers, feats, values, _ = _scene(cuda, 20, 1)
    g = torch.Generator().manual_seed(2)
    dims = [32, 64, 64, 64, 64, 4]
    params = []
    for a, b in zip(dims[:-1], dims[1:]):
        params += [torch.randn(b, a, generator=g).to(cuda), torch.zeros(b, device=cuda)]
    idx, xyz, dists, depths = _rows(cuda, 5, 8, 20, vs, centers, 3)
    assert not train._batch_ok(values, params, idx, xyz, dists, depths, centers, feats)
    out = train.RayChunk.apply(values, *params, idx, xyz, dists, depths, centers, feats, vs, False)
    assert out[0].shape == (5, 3)


@pytest.mark.parametrize("n_vox,bits,rule", [(3, 4, 1), (40, 8, 1), (301, 8, 0), (9, 16, 0),
                                             (500, 2, 1), (77, 5, 0)])
def test_prune_fp32_stage_keeps_the_mask(cuda, n_vox, bits, rule):
    """prune_mask with its FP32 stage against float64 torch at every point,
    thresholds through the middle of the voxels' scores, so that many points
    are close. A wide band sends most points through the FP32 stage."""
    from nsvf_gb300 import ext, geometry
    from nsvf_gb300.field import StandInField
    from nsvf_gb300.mlp import TensorCoreMLP
    vs, centers, feats, values, params = _scene(cuda, n_vox, n_vox)
    field = StandInField(weights=[(params[2 * l].cpu(), params[2 * l + 1].cpu())
                                  for l in range(5)]).to(cuda)
    mlp = TensorCoreMLP(field)
    pts = geometry.offset_points(centers, torch.tensor(vs / 2.0, device=cuda), bits=bits)
    idx = torch.arange(n_vox, device=cuda)[:, None].expand(*pts.shape[:2])
    _, x = _field64(idx, pts.double(), centers.double(), feats, values.double(),
                    [p.double() for p in params], float(np.float32(vs)))
    top = x[:, 0].reshape(n_vox, -1).max(1)[0]
    T = float(top[top > 0].median()) * (1 + 1e-9)
    step = 0.01 if rule else 0.0
    th = -np.expm1(-T * (step if rule else 1.0))
    want = top >= T
    for band in (0.02, 0.5):
        keep, _, n = mlp.prune_mask(centers, feats, values, vs, th=th, bits=bits, rule=rule,
                                    step=step, band=band)
        ext.check_errors(cuda)
        assert torch.equal(keep, want) and n > 0
        # a few points of every voxel first, then the rest's
        keep2, none, _ = mlp.prune_mask(centers, feats, values, vs, th=th, bits=bits, rule=rule,
                                        step=step, band=band, scores=False)
        ext.check_errors(cuda)
        assert torch.equal(keep2, want) and none is None


@pytest.mark.parametrize("n_vox,bits", [(60, 3), (60, 4), (60, 7), (6, 40), (6, 41)])
def test_prune_in_parts_keeps_the_mask(cuda, n_vox, bits):
    """The screen of all points at the edges of its rule (four parts from 4 to
    40 points per axis), and where the parts do not divide the points: the
    mask of the screen in one pass over all points."""
    from nsvf_gb300 import ext
    from nsvf_gb300.field import StandInField
    from nsvf_gb300.mlp import TensorCoreMLP
    vs, centers, feats, values, params = _scene(cuda, n_vox, n_vox)
    mlp = TensorCoreMLP(StandInField(weights=[(params[2 * l].cpu(), params[2 * l + 1].cpu())
                                              for l in range(5)]).to(cuda))
    score = mlp.prune_scores(centers, feats, values, vs, bits=bits, rule=1, step=0.01)
    for th in (float(score.median()), float(score.max()) * 0.999):
        keep = [mlp.prune_mask(centers, feats, values, vs, th=max(th, 1e-6), bits=bits, rule=1,
                               step=0.01, band=band, scores=s)[0]
                for band in (0.02, 0.5) for s in (True, False)]
        ext.check_errors(cuda)
        assert all(torch.equal(k, keep[0]) for k in keep)


@pytest.mark.parametrize("ns", [1, 7, 257, 90001])
@pytest.mark.parametrize("E,dtypes", [(4, (torch.int64, torch.int64)),
                                      (32, (torch.int64, torch.int64)),
                                      (32, (torch.int32, torch.int32)),
                                      (128, (torch.int32, torch.int64))])
def test_interpolation_runs(cuda, ns, E, dtypes):
    """trilinear_embed forward and backward, the kernels for 32 channels (4
    samples per group of lanes) and the general ones: runs of samples in one
    voxel longer and shorter than a group, voxel and corner ids out of range:
    against float64 torch."""
    from nsvf_gb300 import ext
    from nsvf_gb300.functional import trilinear_embed
    n_vox = 50
    vs, centers, feats, _, _ = _scene(cuda, n_vox, E)
    g = torch.Generator().manual_seed(ns + E)
    values = torch.randn(3 * n_vox, E, generator=g).to(cuda).requires_grad_(True)
    lens = torch.randint(1, 40, (ns,), generator=g)
    vid = torch.randint(0, n_vox, (ns,), generator=g).repeat_interleave(lens)[:ns]
    bad = torch.rand(ns, generator=g) < 0.02
    vid = torch.where(bad, torch.where(torch.rand(ns, generator=g) < 0.5, -1, n_vox), vid)
    feats = feats.clone()
    feats[7, 3], feats[9, 0] = -1, 3 * n_vox
    vid, feats, bad = vid.to(cuda), feats.to(dtypes[1]), bad.to(cuda)
    xyz = centers[vid.clamp(0, n_vox - 1)] + (torch.rand(ns, 3, generator=g).to(cuda) - 0.5) * vs
    xyz = xyz.requires_grad_(True)
    gr = torch.randn(ns, E, generator=g).to(cuda)
    ext.error_word(cuda).zero_()
    emb = trilinear_embed(vid.to(dtypes[0]), xyz, centers, feats, values, vs)
    gx, gv = torch.autograd.grad(emb, (xyz, values), gr)
    flagged = int(ext.error_word(cuda).item())
    ext.error_word(cuda).zero_()
    v = vid.clamp(0, n_vox - 1)
    assert flagged == (4 if bad.any() or ((v == 7) | (v == 9)).any() else 0)
    x64, v64 = xyz.detach().double().requires_grad_(True), values.detach().double().requires_grad_(True)
    p = (x64 - centers[v].double()) / vs + 0.5
    ref = 0
    for k in range(8):
        w = 1
        for d, bit in enumerate((4, 2, 1)):
            w = w * (p[:, d] if k & bit else 1 - p[:, d])
        key = feats[v, k].long()
        ok = ((key >= 0) & (key < values.size(0)) & ~bad).double()
        ref = ref + (w * ok)[:, None] * v64[key.clamp(0, values.size(0) - 1)]
    rx, rv = torch.autograd.grad(ref, (x64, v64), gr.double())
    # 8 products of order 1; gradients: a sum over the channels times 1 / vs,
    # and over up to ns / 150 * 8 samples per corner row
    assert float((emb.detach().double() - ref.detach()).abs().max()) <= 1e-5
    assert float((gx.double() - rx).norm()) <= 2e-6 * float(rx.norm()) + 1e-12
    assert float((gv.double() - rv).norm()) <= 2e-6 * float(rv.norm()) + 1e-12


@pytest.mark.parametrize("ns", [128, 152 * 128 * 3 + 1])
def test_head_gradient_of_uneven_quarters(cuda, ns):
    """dW4 where the four threads that hold a sample's last activations find
    largest elements far apart (units of one quarter scaled by 2^20 and the
    head's columns by 2^-20, which leaves the field as it is): all of them have
    to divide by the power of two that is stored beside the row. Against float64
    with the test above's 2^-18 of a column block's norm, and the same bits from
    every launch (each block has several tiles at the larger size)."""
    from nsvf_gb300.functional import trilinear_embed
    from nsvf_gb300 import ext, train
    from nsvf_gb300._lib import LIB, check
    n_vox = 61
    vs, centers, feats, values, params = _scene(cuda, n_vox, 4)
    for q, scale in enumerate((1.0, 2.0 ** 20, 2.0 ** -20, 2.0 ** 10)):
        u = slice(32 * q, 32 * q + 32)
        params[6][u] *= scale
        params[7][u] *= scale
        params[8][:, u] /= scale
    g = torch.Generator().manual_seed(ns)
    vid = torch.randint(0, n_vox, (ns,), generator=g, dtype=torch.int32).to(cuda)
    xyz = (centers[vid.long()] + (torch.rand(ns, 3, generator=g).to(cuda) - 0.5) * vs).contiguous()
    xyzd = torch.cat([xyz, torch.ones(ns, 1, device=cuda)], 1).contiguous()
    dout = torch.randn(ns, 4, generator=g).to(cuda)
    stream, err = ext.ctypes_stream(cuda), ext.error_word(cuda)
    packed = train.RayBatch._packed(params, stream)
    out = torch.empty(ns, 4, device=cuda)
    signs = torch.zeros(4, ns, 16, dtype=torch.uint8, device=cuda)
    scene = (n_vox, values.size(0), vs, centers.data_ptr(), feats.data_ptr(), values.data_ptr(),
             packed.data_ptr())
    check(LIB.nsvf_field_train_forward_signs(ns, vid.data_ptr(), xyzd.data_ptr(), *scene,
                                             out.data_ptr(), signs.data_ptr(), err.data_ptr(),
                                             stream), "forward")
    chunk = -(-ns // 128) * 128
    n = int(LIB.nsvf_field_train_backward_floats(ns, chunk))
    work = torch.empty(n, device=cuda)
    first = None
    for _ in range(10):
        gv, grads = torch.zeros_like(values), [torch.empty_like(p) for p in params]
        check(LIB.nsvf_field_train_backward(
            ns, chunk, vid.data_ptr(), xyzd.data_ptr(), *scene, signs.data_ptr(), dout.data_ptr(),
            work.data_ptr(), n, gv.data_ptr(), train._ptrs(grads[0::2]), train._ptrs(grads[1::2]),
            err.data_ptr(), stream), "backward")
        first = first or grads
        assert all(torch.equal(a, b) for a, b in zip(grads, first))
    ext.check_errors(cuda)
    x = trilinear_embed(vid, xyz, centers, feats, values, vs)
    x64 = x.double()
    for l in range(4):
        z = torch.addmm(params[2 * l + 1], x, params[2 * l].t())
        x64 = (x64 @ params[2 * l].double().t() + params[2 * l + 1].double()) * (z > 0)
        x = torch.relu(z)
    ref = dout.double().t() @ x64
    for q in range(4):
        a, b = first[8][:, 32 * q:32 * q + 32].double(), ref[:, 32 * q:32 * q + 32]
        assert float((a - b).norm()) <= 2.0 ** -18 * float(b.norm())


@pytest.mark.parametrize("units", [0, 12])
@pytest.mark.parametrize("ns,large", [(1, []), (127, [5]), (128, [5, 70]), (129, [128]), (300, [7])])
def test_small_elements_of_the_gradients(cuda, ns, large, units):
    """Single elements: of units that are active only in samples whose
    gradients are 1e-6 of the largest, and of layers whose units differ by 2^24
    in size (scaled by powers of two, which leaves the field as it is). Against
    float64 with the forward's ReLU signs, each element relative to the sum of
    its terms' absolute values: at most six contractions of 128 or ns terms in
    FP32, each a random walk of 2^-24 a term whose largest of 1e5 elements is
    4.5 deviations: 2^-17.5, with a factor of 3 left 2^-16."""
    g = torch.Generator().manual_seed(ns + units)
    dout = torch.randn(ns, 4, generator=g)
    dout[large] *= 1e6
    dout = dout.to(cuda)

    def rescale(params):
        for l in range(4):
            s = 2.0 ** (units * torch.randint(-1, 2, (128,), generator=g).float()).to(cuda)
            params[2 * l] *= s[:, None]
            params[2 * l + 1] *= s
            params[2 * l + 2] /= s

    (grads, gv), (acts, pre, params, scene) = _field_grads(cuda, ns, dout, ns, 304 * 128,
                                                           rescale=rescale)
    vid, xyz, centers, feats, values, vs = scene
    p64 = [p.double() for p in params]
    q = (xyz.double() - centers[vid.long()].double()) / float(np.float32(vs)) + 0.5
    w = [1, 1, 1, 1, 1, 1, 1, 1]
    for k in range(8):
        for d, bit in enumerate((4, 2, 1)):
            w[k] = w[k] * (q[:, d] if k & bit else 1 - q[:, d])
    keys = feats[vid.long()].long()
    v64 = values.double()
    a = [sum(w[k][:, None] * v64[keys[:, k]] for k in range(8))]
    size = [sum(w[k].abs()[:, None] * v64[keys[:, k]].abs() for k in range(8))]
    for l in range(4):
        on = (pre[l] > 0).double()
        a.append((a[-1] @ p64[2 * l].t() + p64[2 * l + 1]) * on)
        size.append((size[-1] @ p64[2 * l].abs().t() + p64[2 * l + 1].abs()) * on)
    ref, da = _chain_grads(a, pre, p64, dout.double())
    sizes, dsize = _chain_grads(size, pre, [p.abs() for p in p64], dout.double().abs())
    ref_v, size_v = (torch.zeros_like(v64) for _ in range(2))
    for k in range(8):
        ref_v.index_add_(0, keys[:, k], w[k][:, None] * da)
        size_v.index_add_(0, keys[:, k], w[k].abs()[:, None] * dsize)
    for x, b, s in zip([*grads, gv], [*ref, ref_v], [*sizes, size_v]):
        assert bool(((x.double() - b).abs() <= 2.0 ** -16 * s).all())


@pytest.mark.parametrize("ns,chunk", [(100000, 640), (1700000, 5 * 304 * 128)])
def test_weight_chains_of_several_sets(cuda, ns, chunk):
    """Gradients where the FP32 chains begin anew on the way (chunks of few
    tiles; more samples than one set takes): at most 9,216 additions round in a
    chain, as a random walk by 2^-24 each: 2^-17 of the norm."""
    from nsvf_gb300._lib import LIB
    assert LIB.nsvf_field_train_chain_chunks(ns, chunk) < -(-ns // chunk)
    g = torch.Generator().manual_seed(ns)
    dout = torch.randn(ns, 4, generator=g).to(cuda)
    (grads, _), (acts, pre, params, _) = _field_grads(cuda, ns, dout, ns, chunk)
    p64 = [p.double() for p in params]
    ref = [0] * 10
    for i in range(0, ns, 250000):
        s = slice(i, i + 250000)
        part, _ = _chain_grads([a[s].double() for a in acts], [z[s] for z in pre], p64,
                               dout[s].double())
        ref = [r + q for r, q in zip(ref, part)]
    for a, b in zip(grads, ref):
        assert float((a.double() - b).norm()) <= 2.0 ** -17 * float(b.norm())


@pytest.mark.parametrize("rays,steps", [(1, 1), (200, 40)])
def test_gradients_behind_a_wait_that_ran_out_are_nan(cuda, rays, steps):
    """A wait of the backward that runs out records bit 3 (8) in the error word
    and leaves partial sums. Set by hand here: every gradient is NaN, so that no
    optimizer takes them for gradients, and the word still says why; without
    it the same call gives finite ones."""
    from nsvf_gb300 import ext, train
    vs, centers, feats, values, params = _scene(cuda, 20, 1)
    idx, xyz, dists, depths = _rows(cuda, rays, steps, 20, vs, centers, 3)
    idx[0, 0] = 4
    values.requires_grad_(True)
    for p in params:
        p.requires_grad_(True)
    word = ext.error_word(cuda)
    for bits in (8, 0):
        word.zero_()
        out = train.RayBatch.apply(values, *params, idx, xyz, dists, depths, centers, feats, vs,
                                   False, 1024)
        word.fill_(bits)
        grads = torch.autograd.grad(out[0].sum(), [values, *params])
        assert int(word.item()) == bits
        word.zero_()
        for g in grads:
            assert bool(g.isnan().all()) if bits else bool(g.isfinite().all())


@pytest.mark.parametrize("n_vox,bits", [(5, 3), (5, 4), (3, 12), (2, 41)])
def test_undecided_points_are_listed_once(cuda, n_vox, bits):
    """With a band that leaves every point undecided: each point once, whether
    the screen goes over all points at once, or over a few of every voxel first
    and the rest in parts; and no other mask than the narrow band's."""
    from nsvf_gb300 import ext
    from nsvf_gb300.field import StandInField
    from nsvf_gb300.mlp import TensorCoreMLP
    vs, centers, feats, values, params = _scene(cuda, n_vox, n_vox)
    params[7] += 1.0                   # active units at every point: M > 0
    mlp = TensorCoreMLP(StandInField(weights=[(params[2 * l].cpu(), params[2 * l + 1].cpu())
                                              for l in range(5)]).to(cuda))
    score = mlp.prune_scores(centers, feats, values, vs, bits=bits, rule=1, step=0.01)
    th = max(float(score.median()), 1e-6)
    want = mlp.prune_mask(centers, feats, values, vs, th=th, bits=bits, rule=1, step=0.01)[0]
    for scores in (True, False):
        keep, _, n = mlp.prune_mask(centers, feats, values, vs, th=th, bits=bits, rule=1,
                                    step=0.01, band=1e6, scores=scores)
        ext.check_errors(cuda)
        assert n == n_vox * bits ** 3
        assert torch.equal(keep, want)


@pytest.mark.parametrize("n_vox,bits", [(65535, 4), (65536, 4), (12300, 7), (66, 40), (62, 41)])
def test_prune_of_many_points_in_parts_keeps_the_mask(cuda, n_vox, bits):
    """From 4 M points on the screen of all points goes in four parts (4 to 40
    points per axis): the mask of the screen in one pass, with undecided points
    on both sides of the number from which FP32 comes before double-float."""
    from nsvf_gb300 import ext
    from nsvf_gb300.field import StandInField
    from nsvf_gb300.mlp import TensorCoreMLP
    vs, centers, feats, values, params = _scene(cuda, n_vox, n_vox)
    mlp = TensorCoreMLP(StandInField(weights=[(params[2 * l].cpu(), params[2 * l + 1].cpu())
                                              for l in range(5)]).to(cuda))
    score = mlp.prune_scores(centers, feats, values, vs, bits=bits, rule=1, step=0.01)
    seen = []
    for th in (float(score.median()), float(score.max()) * 0.999):
        keep = []
        for band in (0.02, 1e-4):
            for s in (True, False):
                k, _, n = mlp.prune_mask(centers, feats, values, vs, th=max(th, 1e-6), bits=bits,
                                         rule=1, step=0.01, band=band, scores=s)
                keep.append(k)
                seen.append(n > mlp.FP32_FROM)
            assert torch.equal(keep[-1], keep[-2])
        ext.check_errors(cuda)
    assert any(seen) and not all(seen)
