"""The workloads that a user of this framework runs, through its public entry
points, for timing and for comparing results.

The path is sparse-voxel rendering: rays are intersected with a voxel set,
samples are placed inside the hit intervals, voxel-corner embeddings are
interpolated there, a 4 x 128 field gives density and colour, and the samples
are composited; training differentiates it, pruning drops empty voxels. The
cases are the operators of that path one by one, the differentiable blocks
forward and backward, and three whole calls (a served frame, a small served
frame, a training step). Scenes, cameras and fields follow the repository's
own workloads: the voxelised shell of a sphere and a torus in [-1, 1]^3
(voxel 1/n, 1/64 at the largest: about 125,000 voxels), cameras on a sphere
of radius 4 looking at the origin, 32 channels per voxel corner, step
voxel / 8. The cameras and rays, the embeddings, the jitter and (except for
pruning, whose field has to reach the threshold) the field's weights come from
the seed.

Each case is a dict with "kind" and its sizes:

* n      voxels per unit length (voxel size 1/n)
* rays   rays of the call, or "size" for a size x size frame
* hits   hit slots per ray (max_hits)
"""
import argparse
import math

import torch

from nsvf_gb300 import clib, ext, functional, scenes, served, train
from nsvf_gb300.encoder import SparseVoxelEncoder
from nsvf_gb300.field import StandInField
from nsvf_gb300.mlp import TensorCoreMLP

EMBED = 32
MLP_FLOPS = 107520.0            # 2 (32 128 + 3 128 128 + 128 4) per sample
SIGMA_SCALE = 7.0               # the renderer's free energy is relu(sigma) dist 7


def listed():
    return [
        # A full frame of the largest scene, as the render server produces it.
        {"name": "frame_800", "kind": "frame", "n": 64, "size": 800, "hits": 64},
        # The smallest frame: a 64 x 64 preview of a 0.25-voxel ball, latency.
        {"name": "frame_64", "kind": "frame", "n": 4, "size": 64, "hits": 20},
        # One training iteration, 4 views x 2,048 rays: intersection, samples,
        # loss, gradients of the embeddings and the field.
        {"name": "train_step", "kind": "train", "n": 64, "rays": 8192, "hits": 64},
        # Its differentiable part alone on given samples, with the colours'
        # gradient from the user's own loss.
        {"name": "render_grad", "kind": "render", "n": 64, "rays": 8192},
        # The octree traversal operator on a frame of rays.
        {"name": "svo_frame", "kind": "svo", "n": 64, "rays": 640000, "hits": 64},
        # The brute-force operator on a training batch while the voxels are
        # still coarse (the encoder's path without an octree).
        {"name": "aabb_batch", "kind": "aabb", "n": 16, "rays": 8192, "hits": 60},
        # Sample placement for a training batch, random jitter.
        {"name": "cdf_batch", "kind": "cdf", "n": 64, "rays": 8192, "hits": 64, "jitter": True},
        # Sample placement for the hit rays of a frame, no jitter.
        {"name": "cdf_frame", "kind": "cdf", "n": 64, "rays": 120000, "hits": 64, "jitter": False},
        # The uniform sampler on a 64 x 64 view's hit rays.
        {"name": "uniform_view", "kind": "uniform", "n": 4, "rays": 1070, "hits": 20,
         "jitter": True},
        # Interpolation of a batch of samples, forward and backward (to the
        # embeddings and, as the encoder asks for it, the positions).
        {"name": "interp_grad", "kind": "interp", "n": 64, "samples": 1260858},
        # Compositing of a training batch, forward and backward.
        {"name": "composite_grad", "kind": "composite", "rays": 8192, "steps": 400},
        # Self-pruning of the largest scene, the exact mask.
        {"name": "prune", "kind": "prune", "n": 64, "bits": 8, "use_step": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame", "train", "render", "svo", "aabb", "cdf", "uniform", "interp",
                       "composite", "prune"])
    hits = rng.choice([20, 33, 60, 64])
    if kind == "frame":
        return {"kind": kind, "n": _log_int(rng, 4, 64), "size": _log_int(rng, 64, 790),
                "hits": hits}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 12, 64), "rays": _log_int(rng, 512, 8000),
                "hits": hits}
    if kind == "render":
        return {"kind": kind, "n": _log_int(rng, 12, 64), "rays": _log_int(rng, 512, 8000)}
    if kind == "svo":
        return {"kind": kind, "n": _log_int(rng, 4, 64), "rays": _log_int(rng, 4096, 600000),
                "hits": hits}
    if kind == "aabb":
        return {"kind": kind, "n": _log_int(rng, 4, 16), "rays": _log_int(rng, 1024, 8000),
                "hits": hits}
    if kind == "cdf":
        jitter = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 4, 64),
                "rays": _log_int(rng, 1000, 30000 if jitter else 115000), "hits": hits,
                "jitter": jitter}
    if kind == "uniform":
        return {"kind": kind, "n": _log_int(rng, 4, 32), "rays": _log_int(rng, 1000, 8192),
                "hits": hits, "jitter": rng.random() < 0.5}
    if kind == "interp":
        return {"kind": kind, "n": _log_int(rng, 12, 64), "samples": _log_int(rng, 20000, 1200000)}
    if kind == "composite":
        return {"kind": kind, "rays": _log_int(rng, 1024, 8000), "steps": _log_int(rng, 40, 390)}
    use_step = rng.random() < 0.5
    return {"kind": "prune", "n": _log_int(rng, 8, 60 if use_step else 20),
            "bits": 8 if use_step else 16, "use_step": use_step}


# ------------------------------------------------------------------ scenes --

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _grid(n):
    """Integer cells [-n, n]^3 whose centres i / n fill [-1, 1]^3."""
    i = torch.arange(-n, n + 1, device="cuda")
    return torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3)


def _voxels(n):
    """(cells [V, 3] int64, centres [V, 3] FP32): at n < 12 the ball of radius
    0.8, else the shell |SDF| < 2 voxels of a sphere and a torus."""
    cells = _grid(n)
    c = cells.double() / n
    if n < 12:
        keep = c.norm(dim=-1) <= 0.8
    else:
        sphere = c.norm(dim=-1) - 0.6
        ring = (c[:, 0] ** 2 + c[:, 1] ** 2).sqrt() - 0.7
        torus = (ring ** 2 + c[:, 2] ** 2).sqrt() - 0.2
        keep = torch.minimum(sphere, torus).abs() < 2.0 / n
    cells = cells[keep]
    return cells, (cells.double() / n).float()


def _encoder(points, n, hits, seed, embed=EMBED):
    args = argparse.Namespace(voxel_size=1.0 / n, max_hits=hits, raymarching_stepsize_ratio=0.125,
                              voxel_embed_dim=embed, use_octree=True, deterministic_step=True)
    enc = SparseVoxelEncoder(args, points=points).to(_device())
    with torch.no_grad():
        w = enc.values.weight
        w.copy_(0.01 * torch.randn(w.shape, generator=_gen(seed, 2), device="cuda"))
    return enc


def _field(seed, sigma_scale=1.0, sigma_bias=0.0):
    return StandInField(weights=scenes.stand_in_mlp_weights(
        seed=2 + int(seed) % 1000003, sigma_scale=sigma_scale, sigma_bias=sigma_bias)).to(_device())


def _camera(seed, salt=3):
    v = _uniform(_gen(seed, salt), 3) - 0.5
    return 4.0 * v / v.norm()


def _frame_rays(cam, height, width, focal):
    """Unit directions [height * width, 3] FP32 through the pixel centres of a
    pinhole camera at `cam` that looks at the origin."""
    f = -cam / cam.norm()
    up = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
    r = torch.linalg.cross(f, up)
    r = r / r.norm()
    d = torch.linalg.cross(f, r)
    j = (torch.arange(width, device="cuda").double() + 0.5 - width / 2.0) / focal
    i = (torch.arange(height, device="cuda").double() + 0.5 - height / 2.0) / focal
    rays = (f + j[None, :, None] * r + i[:, None, None] * d).reshape(-1, 3)
    return (rays / rays.norm(dim=-1, keepdim=True)).float()


def _view_rays(rays, seed):
    """`rays` rays of one view of about a square: (origins, directions [R, 3])."""
    h = max(1, int(math.sqrt(rays)))
    w = -(-rays // h)
    cam = _camera(seed)
    rd = _frame_rays(cam, h, w, 1.25 * w)[:rays].contiguous()
    return cam.float().expand(rays, 3).contiguous(), rd


def _hit_rays(points, n, rays, seed):
    """`rays` rays from 4 cameras, each through a random point of a random
    voxel, in view order: (origins, directions [R, 3] FP32)."""
    g = _gen(seed, 4)
    cams = torch.stack([_camera(seed, 10 + k) for k in range(4)])
    view = torch.arange(rays, device="cuda") * 4 // rays
    vox = torch.randint(0, points.size(0), (rays,), generator=g, device="cuda")
    to = points[vox].double() + (_uniform(g, rays, 3) - 0.5) * (0.98 / n)
    d = to - cams[view]
    return cams[view].float().contiguous(), (d / d.norm(dim=-1, keepdim=True)).float().contiguous()


def _march(cells, n, ro, rd):
    """Samples every voxel / 8 along the rays, those inside a voxel packed to
    the front of each row: (voxel ids [R, M] int32 with -1, depths, distances,
    positions [R, M, 3])."""
    side = 2 * n + 1
    ids = torch.full((side ** 3,), -1, dtype=torch.int32, device="cuda")
    flat = ((cells + n) * torch.tensor([side * side, side, 1], device="cuda")).sum(-1)
    ids[flat] = torch.arange(cells.size(0), dtype=torch.int32, device="cuda")
    step = 0.125 / n
    t = torch.arange(int(3.8 / step), device="cuda").float() * step + 2.1
    out = []
    for a in range(0, ro.size(0), 2048):
        x = ro[a:a + 2048, None] + rd[a:a + 2048, None] * t[:, None]
        cell = (x * n).round().long() + n
        inside = ((cell >= 0) & (cell < side)).all(-1)
        cell = cell.clamp(0, side - 1)
        vid = ids[(cell[..., 0] * side + cell[..., 1]) * side + cell[..., 2]]
        vid = vid.masked_fill(~inside, -1)
        hit = vid.ne(-1)
        order = (~hit).to(torch.uint8).sort(dim=1, stable=True)[1]
        m = int(hit.sum(1).max())
        order = order[:, :m]
        out.append((vid.gather(1, order), torch.where(hit.gather(1, order), t[order], 1e4)))
    m = max(v.size(1) for v, _ in out)
    vid = torch.cat([torch.nn.functional.pad(v, (0, m - v.size(1)), value=-1) for v, _ in out])
    dep = torch.cat([torch.nn.functional.pad(d, (0, m - d.size(1)), value=1e4) for _, d in out])
    dist = torch.where(vid.ne(-1), step, 0.0).float()
    return vid, dep, dist, (ro[:, None] + rd[:, None] * dep[..., None]).contiguous()


def _hit_lists(points, n, rays, hits, seed, uniform):
    """Sorted hit lists [R, hits] of hit rays and their distribution. The
    operators' output width is the longest row's number of samples: row 0 is
    the same longest chain of voxels whatever the seed."""
    enc = _encoder(points, n, hits, seed, embed=4)
    ro, rd = _hit_rays(points, n, rays + rays // 4 + 64, seed)
    st = {k: v.unsqueeze(0) for k, v in enc.precompute().items()}
    _, _, inter, _ = enc.ray_intersect(ro[None, None], rd[None, None], st)
    idx, lo, hi = (inter[k][0] for k in ("intersected_voxel_idx", "min_depth", "max_depth"))
    step = float(enc.step_size)
    chain = 32 if n >= 12 and hits >= 32 else 16 if n > 5 else 8
    most = min(512, 20 * n) if uniform else 256 if n >= 12 else 8 * chain
    steps = ext.ray_probs(idx, lo, hi, step)[1]
    # a voxel adds a sample at its exit, and to the uniform sampler's steps
    # (whose jitter is per step of the whole ray) up to two more
    count = steps.ceil() + (3 if uniform else 1) * idx.ne(-1).sum(-1)
    short = (count < most + chain - 2).nonzero()[:, 0]
    rows = short[torch.arange(rays - 1, device="cuda") % short.numel()]
    edge = 3.0 + torch.arange(chain + 1, device="cuda").float() * (most * step / chain)
    pad = (0, hits - chain)
    idx = torch.cat([torch.nn.functional.pad(
        torch.arange(chain, dtype=torch.int32, device="cuda"), pad, value=-1)[None], idx[rows]])
    lo, hi = (torch.cat([torch.nn.functional.pad(e, pad, value=10000.0)[None], d[rows]])
              for e, d in ((edge[:-1], lo), (edge[1:], hi)))
    return (idx, lo, hi, *ext.ray_probs(idx, lo, hi, step))


# ----------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    s = {"kind": kind}
    if kind == "composite":
        return _prepare_composite(case, seed)
    cells, points = _voxels(n)
    if kind == "frame":
        enc = _encoder(points, n, case["hits"], seed).eval()
        s["scene"] = served.SceneState(enc, _field(seed))
        cam = _camera(seed)
        s["ro"] = cam.float()
        s["rd"] = _frame_rays(cam, case["size"], case["size"], 1.25 * case["size"])
    elif kind in ("train", "render"):
        enc = s["enc"] = _encoder(points, n, case.get("hits", 64), seed)
        field = s["field"] = _field(seed, sigma_scale=30.0, sigma_bias=0.5)
        s["params"] = [enc.values.weight] + [p for lin in field.layers
                                             for p in (lin.weight, lin.bias)]
        s["states"] = enc.precompute(id=None)
        s["ro"], s["rd"] = _hit_rays(points, n, case["rays"], seed)
        g = _gen(seed, 5)
        if kind == "train":
            s["target"] = _uniform(g, case["rays"], 3).float()
        else:
            vid, dep, dist, xyz = _march(cells, n, s["ro"], s["rd"])
            hits = vid[:, 0].ne(-1)
            s["samples"] = (hits, vid[hits], dep[hits], dist[hits], xyz[hits])
            s["grad"] = torch.randn(case["rays"], 3, generator=g, device="cuda")
    elif kind == "svo":
        enc = _encoder(points, n, case["hits"], seed, embed=4)
        st = enc.precompute(id=None)
        s["centers"] = st["voxel_octree_center_xyz"][None].contiguous()
        s["children"] = st["voxel_octree_children_idx"][None].contiguous()
        ro, rd = _view_rays(case["rays"], seed)
        s.update(ro=ro[None], rd=rd[None], vs=1.0 / n, hits=case["hits"])
    elif kind == "aabb":
        ro, rd = _hit_rays(points, n, case["rays"], seed)
        s.update(points=points[None].contiguous(), ro=ro[None], rd=rd[None], vs=1.0 / n,
                 hits=case["hits"])
    elif kind in ("cdf", "uniform"):
        s["lists"] = _hit_lists(points, n, case["rays"], case["hits"], seed, kind == "uniform")
        s.update(jitter=case["jitter"], seed=int(seed), step=0.125 / n)
    elif kind == "interp":
        s.update(_prepare_interp(case, seed, cells, points))
    elif kind == "prune":
        enc = s["enc"] = _encoder(points, n, 64, seed).eval()
        # the density row scaled so that about half of the voxels reach the
        # threshold (a sigma of ln 2 / step, or of ln 2)
        scale = 3.6e5 * n / 64 if case["use_step"] else 703.0
        field = StandInField(weights=scenes.stand_in_mlp_weights(seed=2, sigma_scale=scale))
        s["mlp"] = TensorCoreMLP(field.to(_device()))
        s.update(bits=case["bits"], use_step=case["use_step"])
    return s


def _prepare_interp(case, seed, cells, points):
    n, ns = case["n"], case["samples"]
    enc = _encoder(points, n, 64, seed)
    st = enc.precompute(id=None)
    rays = max(64, ns // 40)
    ro, rd = _hit_rays(points, n, rays, seed)
    vid, _, _, xyz = _march(cells, n, ro, rd)
    live = vid.ne(-1)
    vid, xyz = vid[live], xyz[live]
    rep = -(-ns // vid.numel())
    g = _gen(seed, 6)
    return {"vid": vid.repeat(rep)[:ns].long().contiguous(),
            "xyz": xyz.repeat(rep, 1)[:ns].contiguous().requires_grad_(True),
            "centers": st["voxel_center_xyz"], "feats": st["voxel_vertex_idx"],
            "values": st["voxel_vertex_emb"].detach().clone().requires_grad_(True),
            "grad": torch.randn(ns, EMBED, generator=g, device="cuda"), "vs": 1.0 / n}


def _prepare_composite(case, seed):
    R, M = case["rays"], case["steps"]
    g = _gen(seed, 7)
    # the rows of a batch: between an eighth of the slots and all of them are
    # samples, a few rows are full, the rest is padding
    count = (M * (0.125 + 0.875 * _uniform(g, R) ** 3)).ceil()
    live = torch.arange(M, device="cuda")[None] < count[:, None]
    sigma = 4.0 * torch.randn(R, M, generator=g, device="cuda") + 0.5
    fe = torch.relu(sigma) * (1.0 / 512) * SIGMA_SCALE
    tex = torch.randn(R, M, 3, generator=g, device="cuda")
    dep = 3.0 + torch.arange(M, device="cuda").float() / 512 + _uniform(g, R, 1).float()
    zero = torch.zeros((), device="cuda")
    return {"kind": "composite",
            "fe": torch.where(live, fe, zero).requires_grad_(True),
            "tex": torch.where(live[..., None], tex, zero).requires_grad_(True),
            "depth": torch.where(live, dep, zero + 10000.0),
            "grads": (torch.where(live, dep, zero + 10000.0) * 1e-3,
                      torch.randn(R, generator=g, device="cuda"),
                      torch.randn(R, 3, generator=g, device="cuda"))}


# --------------------------------------------------------------------- run --

def run(s):
    kind = s["kind"]
    if kind == "frame":
        return served.render_frame(s["scene"], s["ro"], s["rd"])
    if kind == "train":
        for p in s["params"]:
            p.grad = None
        loss = train.train_step(s["enc"], s["field"], s["ro"], s["rd"], s["target"],
                                states=s["states"])
        return [loss] + [p.grad for p in s["params"]]
    if kind == "render":
        colors = train.render_batch(s["enc"], s["field"], s["ro"], s["rd"], states=s["states"],
                                    samples=s["samples"])
        return [colors.detach()] + list(torch.autograd.grad(colors, s["params"], s["grad"]))
    if kind == "svo":
        return clib.svo_ray_intersect(s["vs"], s["hits"], s["centers"], s["children"], s["ro"],
                                      s["rd"])
    if kind == "aabb":
        return clib.aabb_ray_intersect(s["vs"], s["hits"], s["points"], s["ro"], s["rd"])
    if kind == "cdf":
        if s["jitter"]:
            torch.cuda.manual_seed(s["seed"])
        return clib.inverse_cdf_sampling(*s["lists"], -1, not s["jitter"])
    if kind == "uniform":
        if s["jitter"]:
            torch.cuda.manual_seed(s["seed"])
        idx, lo, hi, _, _ = s["lists"]
        return clib.uniform_ray_sampling(idx, lo, hi, s["step"], 2.0 * math.sqrt(3.0),
                                         not s["jitter"])
    if kind == "interp":
        emb = functional.trilinear_embed(s["vid"], s["xyz"], s["centers"], s["feats"], s["values"],
                                         s["vs"])
        return [emb.detach()] + list(torch.autograd.grad(emb, (s["xyz"], s["values"]), s["grad"]))
    if kind == "composite":
        probs, depth, missed, colors = functional.composite(s["fe"], s["tex"], s["depth"])
        grads = torch.autograd.grad((probs, missed, colors), (s["fe"], s["tex"]), s["grads"])
        return [probs.detach(), depth.detach(), missed.detach(), colors.detach(), *grads]
    if kind == "prune":
        return s["enc"].pruning_exact(s["mlp"], th=0.5, bits=s["bits"], use_step=s["use_step"],
                                      apply=False)
    raise ValueError(kind)


# -------------------------------------------------------------------- work --

def work(case):
    """Sample and voxel counts are those of the scenes' typical view (a shell
    view: 19 % of a frame's rays hit, 160 samples per hit ray)."""
    kind, n = case["kind"], case.get("n", 0)
    vox = 2.2 * n ** 3 if n < 12 else 30.0 * n * n
    keys = 1.4 * vox
    if kind == "frame":
        rays = float(case["size"]) ** 2
        return {"bytes": rays * (12 + 20) + vox * 48 + keys * 128,
                "flops": MLP_FLOPS * rays * (9.0 if n < 12 else 30.0)}
    if kind in ("train", "render"):
        ns = case["rays"] * 160.0
        return {"bytes": ns * (24 if kind == "render" else 0) + keys * 256 + case["rays"] * 36,
                "flops": 3 * MLP_FLOPS * ns}
    if kind == "svo":
        return {"bytes": case["rays"] * (24.0 + 12 * case["hits"]) + 2.2 * vox * 48,
                "flops": case["rays"] * 40.0 * 18}
    if kind == "aabb":
        return {"bytes": case["rays"] * (24.0 + 12 * case["hits"]) + vox * 12,
                "flops": case["rays"] * vox * 18.0}
    if kind == "cdf":
        # the widest row has about 2.5 times the mean row's samples
        return {"bytes": case["rays"] * (16.0 * case["hits"] + 12 * 400 +
                                         (1600 if case["jitter"] else 0)), "flops": 0}
    if kind == "uniform":
        return {"bytes": case["rays"] * (12.0 * case["hits"] + 12 * 60), "flops": 0}
    if kind == "interp":
        ns = float(case["samples"])
        return {"bytes": ns * (8 + 12 + 2 * 128 + 12) + keys * 256 + vox * 76,
                "flops": ns * (8 * EMBED * 6 + 60)}
    if kind == "composite":
        return {"bytes": case["rays"] * (case["steps"] * 44.0 + 40),
                "flops": case["rays"] * case["steps"] * 60.0}
    return {"bytes": vox * 77 + keys * 128, "flops": MLP_FLOPS * vox * case["bits"] ** 3}


# ------------------------------------------------------------------- exact --

def exact(case, seed):
    """Results in 64 bits. Sample placement, the octree and whole calls have
    none: their values follow from FP32 decisions (which cell, which bin) that
    64 bits would take differently."""
    kind = case["kind"]
    if kind == "interp":
        return _exact_interp(prepare(case, seed))
    if kind == "composite":
        s = prepare(case, seed)
        fe, tex = (s[k].detach().double().requires_grad_(True) for k in ("fe", "tex"))
        p, depth, missed, colors = _composite64(fe, tex, s["depth"].double())
        grads = torch.autograd.grad((p, missed, colors), (fe, tex),
                                    [g.double() for g in s["grads"]])
        return [p.detach(), depth.detach(), missed.detach(), colors.detach(), *grads]
    if kind == "render":
        return _exact_render(prepare(case, seed))
    if kind == "aabb":
        return _exact_aabb(prepare(case, seed))
    return None


def _composite64(fe, tex, depth):
    shifted = torch.cat([fe.new_zeros(fe.size(0), 1), fe[:, :-1]], 1)
    p = (1 - torch.exp(-fe)) * torch.exp(-shifted.cumsum(1))
    return p, (p * depth).sum(1), 1 - p.sum(1), (p[..., None] * tex).sum(1)


def _interp64(vid, xyz, centers, feats, values, vs):
    p = (xyz - centers[vid]) / vs + 0.5
    emb = 0
    for k in range(8):
        w = 1
        for d, bit in enumerate((4, 2, 1)):
            w = w * (p[:, d] if k & bit else 1 - p[:, d])
        emb = emb + w[:, None] * values[feats[vid, k]]
    return emb


def _exact_interp(s):
    xyz, values = (s[k].detach().double().requires_grad_(True) for k in ("xyz", "values"))
    emb = _interp64(s["vid"], xyz, s["centers"].double(), s["feats"].long(), values,
                    float(torch.tensor(s["vs"]).float()))
    return [emb.detach(), *torch.autograd.grad(emb, (xyz, values), s["grad"].double())]


def _exact_render(s):
    params = [p.detach().double().requires_grad_(True) for p in s["params"]]
    values, layers = params[0], params[1:]
    hits, vid, dep, dist, xyz = s["samples"]
    centers = s["states"]["voxel_center_xyz"].double()
    feats = s["states"]["voxel_vertex_idx"].long()
    vs = float(s["enc"].voxel_size)
    bg = s["field"].bg_color.bg_color.detach().double()
    colors = bg.expand(hits.numel(), 3).clone()
    rows = hits.nonzero()[:, 0]
    total = [torch.zeros_like(p) for p in params]
    for a in range(0, rows.numel(), 1024):
        b = slice(a, a + 1024)
        mask = vid[b].ne(-1)
        x = _interp64(vid[b][mask].long(), xyz[b][mask].double(), centers, feats, values, vs)
        for i in range(0, len(layers), 2):
            x = x @ layers[i].t() + layers[i + 1]
            x = torch.relu(x) if i + 2 < len(layers) else x
        zero = dist.new_zeros(mask.shape, dtype=torch.float64)
        fe = zero.masked_scatter(mask, torch.relu(x[:, 0]) * dist[b][mask].double() * SIGMA_SCALE)
        tex = torch.stack([zero.masked_scatter(mask, x[:, 1 + c]) for c in range(3)], -1)
        _, _, missed, col = _composite64(fe, tex, dep[b].double())
        col = col + missed[:, None] * bg
        for t, g in zip(total, torch.autograd.grad(col, params, s["grad"][rows[b]].double())):
            t += g
        colors[rows[b]] = col.detach()
    return [colors, *total]


def _exact_aabb(s):
    """Depths of the first `hits` voxels, in voxel order, that each ray's slab
    test in 64 bits finds."""
    c, h, H = s["points"][0].double(), s["vs"] / 2, s["hits"]
    ro, rd = s["ro"][0].double(), s["rd"][0].double()
    out = []
    for a in range(0, ro.size(0), 512):
        lo = ro.new_zeros(ro[a:a + 512].size(0), c.size(0))
        hi = lo + 1e5
        for d in range(3):
            o, inv = ro[a:a + 512, d, None], 1.0 / rd[a:a + 512, d, None]
            t0, t1 = (c[:, d] - h - o) * inv, (c[:, d] + h - o) * inv
            lo = torch.maximum(lo, torch.minimum(t0, t1))
            hi = torch.minimum(hi, torch.maximum(t0, t1))
        hit = lo <= hi
        order = (~hit).to(torch.uint8).sort(dim=1, stable=True)[1][:, :H]
        live = hit.gather(1, order)
        d = [torch.where(live, t.gather(1, order), 0.0) for t in (lo, hi)]
        out.append([torch.nn.functional.pad(t, (0, H - t.size(1))) for t in d])
    return [None, torch.cat([o[0] for o in out])[None], torch.cat([o[1] for o in out])[None]]
