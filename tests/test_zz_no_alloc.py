"""The allocation-free SVO intersection entry point (nsvf_svo_intersect_noalloc).

Some callers cannot allocate device memory while they render: a real-time
loop or a host engine with a fixed, pre-partitioned memory budget that passes
this library only its own input and output buffers. For them the library
keeps the octree scratch in a fixed-size array of its own. This test calls
that entry point through the C ABI, twice in a row, and checks that its
outputs are identical (the op is exact) to the allocating nsvf_svo_intersect
and that the repeat call takes no device memory; that octrees beyond the
fixed scratch are refused; and that it works filled to its capacity.

The file is named so that pytest collects it last.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NOALLOC_MAX_NODES = 1 << 18


def _noalloc_fn():
    from nsvf_gb300._lib import LIB_PATH
    lib = ctypes.CDLL(LIB_PATH)
    fn = lib.nsvf_svo_intersect_noalloc
    P, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    fn.argtypes = [i32, i32, i32, i32, f32, i32, P, P, P, P, P, P, P, P, P]
    fn.restype = i32
    return fn


def _rays(n, seed):
    rng = np.random.RandomState(seed)
    o = rng.normal(size=(n, 3))
    o = 3.0 * o / np.linalg.norm(o, axis=1, keepdims=True)
    d = -o + rng.normal(scale=0.4, size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


def test_noalloc_matches_allocating_entry_point(cuda):
    from nsvf_gb300 import ext, geometry, scenes
    p, vs = scenes.scene_shell(1.0 / 32)
    cen, chi = geometry.build_easy_octree(torch.from_numpy(p), vs / 2)
    n = cen.shape[0]
    assert n <= NOALLOC_MAX_NODES
    cen, chi = cen[None].contiguous().to(cuda), chi[None].contiguous().to(cuda)
    o, d = _rays(5000, seed=3)
    rs = torch.from_numpy(o)[None].to(cuda)
    rd = torch.from_numpy(d)[None].to(cuda)
    H = 64
    ref = ext.svo_intersect(rs, rd, cen, chi, vs, H)
    fn = _noalloc_fn()
    stream = torch.cuda.current_stream(cuda).cuda_stream
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    outs = [(torch.full((1, 5000, H), 7, dtype=torch.int32, device=cuda),
             torch.full((1, 5000, H), 7.0, device=cuda), torch.full((1, 5000, H), 7.0, device=cuda))
            for _ in range(2)]
    free = []
    for idx, lo, hi in outs:
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info(cuda)[0])
        st = fn(1, 1, n, 5000, vs, H, rs.data_ptr(), rd.data_ptr(), cen.data_ptr(), chi.data_ptr(),
                idx.data_ptr(), lo.data_ptr(), hi.data_ptr(), err.data_ptr(), stream)
        assert st == 0
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        assert torch.equal(idx, ref[0])
        assert torch.equal(lo, ref[1])
        assert torch.equal(hi, ref[2])
    # the second call took no device memory (the first may have set up the
    # context's module); outputs were allocated before either call
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info(cuda)[0] == free[1]
    assert int((ref[0] != -1).sum()) > 1000


def test_noalloc_rejects_octrees_beyond_its_scratch(cuda):
    """More than NSVF_NOALLOC_MAX_NODES nodes in all -- one large octree, or
    b_pts point sets whose product of counts exceeds it -- is refused before
    anything is launched."""
    fn = _noalloc_fn()
    dummy = torch.zeros(16, device=cuda)
    p = dummy.data_ptr()
    s = torch.cuda.current_stream(cuda).cuda_stream
    assert fn(1, 1, NOALLOC_MAX_NODES + 1, 4, 0.1, 8, p, p, p, p, p, p, p, None, s) == -4
    half = NOALLOC_MAX_NODES // 2 + 1
    assert fn(2, 2, half, 4, 0.1, 8, p, p, p, p, p, p, p, None, s) == -4


def test_noalloc_at_its_capacity(cuda):
    """b_pts copies of a small octree filling the scratch to within one copy
    of NSVF_NOALLOC_MAX_NODES (176 bytes per node, the root boxes included),
    one ray per copy: the same outputs as the allocating entry point."""
    from nsvf_gb300 import ext, geometry, scenes
    p, vs = scenes.scene_small()
    cen, chi = geometry.build_easy_octree(torch.from_numpy(p), vs / 2)
    n = cen.shape[0]
    b = NOALLOC_MAX_NODES // n
    assert b * n > NOALLOC_MAX_NODES - n
    cen_b = cen[None].expand(b, n, 3).contiguous().to(cuda)
    chi_b = chi[None].expand(b, n, 9).contiguous().to(cuda)
    o, d = _rays(b, seed=5)
    rs = torch.from_numpy(o).reshape(b, 1, 3).to(cuda)
    rd = torch.from_numpy(d).reshape(b, 1, 3).to(cuda)
    H = 20
    ref = ext.svo_intersect(rs, rd, cen_b, chi_b, vs, H)
    idx = torch.empty(b, 1, H, dtype=torch.int32, device=cuda)
    lo, hi = torch.empty(b, 1, H, device=cuda), torch.empty(b, 1, H, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    fn = _noalloc_fn()
    st = fn(b, b, n, 1, vs, H, rs.data_ptr(), rd.data_ptr(), cen_b.data_ptr(), chi_b.data_ptr(),
            idx.data_ptr(), lo.data_ptr(), hi.data_ptr(), err.data_ptr(),
            torch.cuda.current_stream(cuda).cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(idx, ref[0]) and torch.equal(lo, ref[1]) and torch.equal(hi, ref[2])
    assert int((ref[0] != -1).sum()) > 100


def _mixed(seed, sizes):
    from test_ops_gpu import _mixed_tree
    cen, chi = _mixed_tree(seed)
    rng = np.random.RandomState(seed)
    internal = np.flatnonzero(chi[:, 8] > 1)
    leaves = np.flatnonzero(chi[:, 8] == 1)
    n = len(cen)
    if sizes == "two_parents":          # a subtree reached twice
        k = internal[internal < n - 1]
        for a in k[:3]:
            free = [p for p in internal if p > a and (chi[p, :8] == -1).any()]
            p = free[rng.randint(len(free))]
            chi[p, np.flatnonzero(chi[p, :8] == -1)[0]] = a
    elif sizes == "bad_id":
        chi[internal[len(internal) // 2], 3] = n + 5
        chi[internal[0], 1] = -7
    elif sizes == "leaf_children":      # a leaf that lists children
        chi[leaves[1::5], 0] = leaves[0]
        chi[leaves[2::5], 2] = internal[0]
    elif sizes == "nan":
        cen[leaves[::9], 1] = np.nan
        cen[leaves[1::9], 0] = np.inf
    elif sizes == "odd_sizes":          # sizes that are not the tree's
        chi[internal[::3], 8] = 3
        chi[internal[1::7], 8] = -2
        chi[leaves[::11], 8] = 0
    elif sizes == "shifted":            # cubes that do not contain their leaves
        cen[internal[:-1:2]] += rng.uniform(-0.05, 0.05, (len(internal[:-1:2]), 3)).astype(np.float32)
    elif sizes == "cycle":
        p = internal[len(internal) // 2]
        chi[p, 0] = n - 1
    return cen, chi


@pytest.mark.parametrize("form", ["shell", "odd_voxel", "mixed", "two_parents", "bad_id",
                                  "leaf_children", "nan", "odd_sizes", "shifted", "cycle",
                                  "single_leaf", "chain", "chain_center"])
def test_tight_boxes_equal_the_cubes(cuda, form):
    """nsvf_svo_intersect traverses the bounding boxes of the leaves, the
    allocation-free entry point the input's cubes: the same hits and the same
    error bits, for every kind of input table and ray."""
    from nsvf_gb300 import ext, geometry, scenes
    R, H = 3000, 33
    o, d = _rays(R, seed=11)
    rng = np.random.RandomState(1)
    if form in ("shell", "odd_voxel"):
        vs = 1.0 / 32 if form == "shell" else 0.037
        p = scenes.shell_voxels(vs, scenes.sphere_torus_sdf)
        cen, chi = (t.numpy() for t in geometry.build_easy_octree(torch.from_numpy(p), vs / 2))
    elif form == "single_leaf":
        vs, cen, chi = 0.5, np.zeros((1, 3), np.float32), np.array([[-1] * 8 + [1]], np.int32)
    elif form.startswith("chain"):      # 21 levels: deeper than the traversal's stack
        vs, L = 1e-5, 21
        cen = np.zeros((L, 3), np.float32)
        chi = np.full((L, 9), -1, np.int32)
        chi[:, 8] = 2 ** np.arange(L)
        chi[1:, 7] = np.arange(L - 1)
    else:
        vs = 0.04
        cen, chi = _mixed(3, form)
    o[::5] = rng.uniform(-0.3, 0.3, o[::5].shape)            # from inside
    d[::7, 0] = 0.0
    d[1::13] = np.float32([0, 0, -1])
    o[2::9] = np.round(o[2::9] / (vs / 2)) * np.float32(vs / 2)   # on grid planes
    if form == "chain_center":
        d[3::4] = -o[3::4] / np.linalg.norm(o[3::4], axis=1, keepdims=True)
    cen, chi = np.ascontiguousarray(cen, np.float32), np.ascontiguousarray(chi, np.int32)
    t = lambda a: torch.from_numpy(a)[None].contiguous().to(cuda)
    rs, rd, tc, tch = t(o), t(d), t(cen), t(chi)
    ext.error_word(cuda).zero_()
    out = ext.svo_intersect(rs, rd, tc, tch, vs, H)
    srt = ext.svo_intersect_sorted(rs, rd, tc, tch, vs, H)
    got_err = int(ext.error_word(cuda).item())
    ext.error_word(cuda).zero_()
    ref = [torch.empty_like(a) for a in out]
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    status = _noalloc_fn()(1, 1, len(cen), R, vs, H, rs.data_ptr(), rd.data_ptr(), tc.data_ptr(),
                           tch.data_ptr(), *[a.data_ptr() for a in ref], err.data_ptr(),
                           torch.cuda.current_stream(cuda).cuda_stream)
    assert status == 0
    for a, b in zip(out, ref):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert got_err == int(err.item())
    assert (form in ("bad_id", "cycle", "chain_center")) == (got_err != 0)
    if form != "single_leaf" and not form.startswith("chain"):
        assert int(out[0].ne(-1).sum()) > 0
    # the sorted variant: the same rows in depth order, slot order at ties
    m = ref[0].eq(-1)
    lo, order = ref[1].masked_fill(m, 10000.0).sort(dim=-1, stable=True)
    assert torch.equal(srt[1], lo) and torch.equal(srt[0], ref[0].gather(-1, order))
    assert torch.equal(srt[2], ref[2].masked_fill(m, 10000.0).gather(-1, order))
