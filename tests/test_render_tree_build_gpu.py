"""The render tree's build (csrc/render_tree.cu): node for node that of a host PLOC with the same rule, on both sides
of 4,096 clusters, where the rounds move into one block; and frames over the smallest trees against the CPU oracle's, with the
triangles where pixels see them."""
import ctypes as C

import numpy as np
import pytest

import lumina
import oracle as O
from lumina import _ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RADIUS = 8  # places searched on either side


def _area(lo, hi):
    d = hi - lo
    return d[:, 0] * d[:, 1] + d[:, 1] * d[:, 2] + d[:, 2] * d[:, 0]


def host_ploc(lo, hi):
    """Nodes in depth order of PLOC over boxes lo, hi (integers: areas are exact): each cluster's nearest within RADIUS
    places by the area of the union, the lower place among equals; mutual pairs merge at the lower place, numbered in
    order; a stable sort of the nodes by depth."""
    t = len(lo)
    nodes = np.zeros(2 * t - 1, _ffi.NODE_DTYPE)
    nodes["bbMin"][:t], nodes["bbMax"][:t] = lo, hi
    nodes["left"][:t] = nodes["right"][:t] = -1
    nodes["firstTri"][:t] = np.arange(t)
    nodes["triCount"][:t] = 1
    ids, next_id = np.arange(t), t
    while len(ids) > 1:
        c = len(ids)
        best, nn = np.full(c, np.inf), np.full(c, -1)
        for d in [*range(-RADIUS, 0), *range(1, RADIUS + 1)]:
            i = np.arange(max(0, -d), min(c, c - d))
            if len(i) == 0:
                continue
            a = _area(np.minimum(lo[i], lo[i + d]), np.maximum(hi[i], hi[i + d]))
            closer = a < best[i]
            best[i[closer]], nn[i[closer]] = a[closer], (i + d)[closer]
        i = np.arange(c)
        mutual = nn[nn] == i
        own = np.flatnonzero(mutual & (i < nn))
        new = next_id + np.arange(len(own))
        nodes["left"][new], nodes["right"][new] = ids[own], ids[nn[own]]
        lo, hi, ids = lo.copy(), hi.copy(), ids.copy()
        lo[own], hi[own] = np.minimum(lo[own], lo[nn[own]]), np.maximum(hi[own], hi[nn[own]])
        nodes["bbMin"][new], nodes["bbMax"][new] = lo[own], hi[own]
        nodes["firstTri"][new] = -1
        ids[own] = new
        next_id += len(own)
        keep = ~(mutual & (i > nn))
        lo, hi, ids = lo[keep], hi[keep], ids[keep]
    depth = np.zeros(len(nodes), np.int64)
    for k in range(len(nodes) - 1, t - 1, -1):  # a node's number is above its children's
        depth[nodes["left"][k]] = depth[nodes["right"][k]] = depth[k] + 1
    order = np.argsort(depth, kind="stable")
    place = np.empty(len(nodes), np.int32)
    place[order] = np.arange(len(nodes))
    out = nodes[order]
    inner = out["triCount"] == 0
    out["left"][inner], out["right"][inner] = place[out["left"][inner]], place[out["right"][inner]]
    starts = np.searchsorted(depth[order], np.arange(depth.max() + 2))
    return out, starts


def device_ploc(tris):
    """lg::build_render_tree over the triangles, one per leaf: (nodes, first node of each depth)."""
    lib = C.CDLL(str(_ffi.LIB_PATH))
    size = lib._ZN2lg25render_tree_scratch_bytesEii
    size.restype, size.argtypes = C.c_size_t, [C.c_int, C.c_int]
    build = lib._ZN2lg17build_render_treeEPK11lg_bvh_nodeiPK11lg_triangleiiPS0_PiS7_S7_PvmP11CUstream_st
    build.restype = C.c_int
    build.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p,
                      C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
    t, n = len(tris), 2 * len(tris) - 1
    d_tris = torch.from_numpy(tris.view(np.uint8).copy()).cuda()
    d_out = torch.zeros(n * 40, dtype=torch.uint8, device="cuda")
    d_start = torch.zeros(257, dtype=torch.int32, device="cuda")
    start, levels = np.zeros(257, np.int32), C.c_int(0)
    mem = torch.full((size(n, t),), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rc = build(None, n, d_tris.data_ptr(), t, 2, d_out.data_ptr(), d_start.data_ptr(), start.ctypes.data,
               C.addressof(levels), mem.data_ptr(), mem.numel(), torch.cuda.Stream().cuda_stream)
    assert rc == 0
    return d_out.cpu().numpy().view(_ffi.NODE_DTYPE), start[:levels.value + 1]


@pytest.mark.parametrize("t", [2, 3, 33, 4095, 4096, 4097, 9000])
def test_same_tree_as_host_ploc(t):
    """Small boxes with integer corners along a line and around it: many unions of equal area."""
    rng = np.random.default_rng(t)
    at = np.stack([np.arange(t) // 60, rng.integers(0, 12, t), rng.integers(0, 12, t)], -1) + 1
    tris = np.zeros(t, _ffi.TRI_DTYPE)
    tris["v"] = at[:, None, :] + rng.integers(0, 4, (t, 3, 3))
    lo, hi = tris["v"].min(1).astype(np.int64), tris["v"].max(1).astype(np.int64)
    want, want_start = host_ploc(lo, hi)
    got, start = device_ploc(tris)
    assert got.tobytes() == want.tobytes()
    assert (start == want_start).all()


@pytest.mark.parametrize("n", [1, 2, 3, 5])
@pytest.mark.parametrize("tree", ["ploc_tris", "ploc", "buildbvh"])
@pytest.mark.parametrize("width", [2, 4])
def test_smallest_trees_against_oracle(n, tree, width):
    """One to five triangles in front of the camera (1: a leaf is the root; 2: one inner node): the oracle's frame,
    in which they are seen and lit."""
    base = lumina.box_scene(1, width=96, height=48)
    m = np.asarray(base.camera.camera_to_world, np.float32).reshape(4, 4)
    fwd, left, up = m[0, :3], m[1, :3], m[2, :3]
    tris = np.zeros(n, _ffi.TRI_DTYPE)
    for k in range(n):
        c = np.asarray(base.camera.pos, np.float32) + (2.0 + 0.3 * k) * fwd + (0.7 * k - 0.35 * (n - 1)) * left
        tris["v"][k] = [c + 1.2 * left - 1.0 * up, c - 1.2 * left - 1.0 * up, c + 1.2 * up]
        tris["n"][k] = -fwd + 0.5 * up
    tris["n"] /= np.linalg.norm(tris["n"], axis=2, keepdims=True)
    sc = lumina.Scene(base.camera, base.sun, tris, base.mat_albedo, base.mat_emissive, base.points)
    nodes, otris, _, _ = O.oracle_build_bvh(tris)
    want, _ = O.oracle_render(sc, nodes, otris, 4, 1)
    assert (want > 0).any(axis=2).sum() >= 150  # of 4,608 pixels, at most 4 of them differ below
    with lumina.Renderer(0) as r:
        r.set_render_tree(tree)
        r.set_bvh_width(width)
        r.set_scene(sc)
        got = r.render(spp=4, bounces=1)["accum"]
    close = np.abs(got - want) <= 1e-3 * np.maximum(np.abs(want), np.abs(got)) + 1e-6
    assert close.all(axis=2).mean() >= 0.999
