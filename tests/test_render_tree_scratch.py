"""The render tree's scratch holds every tree it is sized for (csrc/render_tree.cu), and the sort's scratch the sort of
any fewer pairs (csrc/radix_sort.cu)."""
import ctypes as C

import numpy as np
import pytest

import lumina
from lumina import _ffi
from test_oracle import soup


def test_sort_scratch_grows_with_n():
    """Scratch sized for n holds the sort of any fewer pairs, whose tiles are smaller and may be more."""
    size = C.CDLL(str(_ffi.LIB_PATH))._ZN2lg24radix_sort_scratch_bytesEm
    size.restype, size.argtypes = C.c_size_t, [C.c_size_t]
    at = sorted({max(1, 148 * t + d) for t in (1, 1024, 2048, 4096, 8192) for d in range(-2, 3)} |
                set(range(1, 2000000, 4099)))
    sizes = [size(n) for n in at]
    assert sizes == sorted(sizes)


def test_sort_refuses_more_pairs_than_bound_for():
    class Scratch(C.Structure):  # lg::RadixSortScratch
        _fields_ = [("pointers", C.c_void_p * 5), ("zero_bytes", C.c_size_t), ("capacity", C.c_size_t),
                    ("poll_limit", C.c_int)]

    sort = C.CDLL(str(_ffi.LIB_PATH))._ZN2lg16radix_sort_pairsEPjS0_miiRKNS_16RadixSortScratchEP11CUstream_stbb
    sort.restype = C.c_int
    sort.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.POINTER(Scratch), C.c_void_p, C.c_bool,
                     C.c_bool]
    s = Scratch(capacity=10)
    assert sort(None, None, 11, 0, 30, C.byref(s), None, True, False) == 1  # cudaErrorInvalidValue, before any launch


def heap_tree(tris, leaves):
    """A complete tree, children of node i at 2 i + 1 and 2 i + 2, of one triangle a leaf and the rest in the last."""
    n = 2 * leaves - 1
    nodes = np.zeros(n, _ffi.NODE_DTYPE)
    lo, hi = tris["v"].min(1), tris["v"].max(1)
    first = leaves - 1
    nodes["left"][:first], nodes["right"][:first] = 2 * np.arange(first) + 1, 2 * np.arange(first) + 2
    nodes["firstTri"][:first] = -1
    nodes["left"][first:] = nodes["right"][first:] = -1
    nodes["firstTri"][first:] = np.arange(leaves)
    nodes["triCount"][first:] = 1
    nodes["triCount"][-1] = len(tris) - leaves + 1
    nodes["bbMin"][first:], nodes["bbMax"][first:] = lo[:leaves], hi[:leaves]
    nodes["bbMin"][-1], nodes["bbMax"][-1] = lo[leaves - 1:].min(0), hi[leaves - 1:].max(0)
    for i in range(first - 1, -1, -1):
        nodes["bbMin"][i] = np.minimum(nodes["bbMin"][2 * i + 1], nodes["bbMin"][2 * i + 2])
        nodes["bbMax"][i] = np.maximum(nodes["bbMax"][2 * i + 1], nodes["bbMax"][2 * i + 2])
    return nodes


@pytest.mark.gpu
def test_scratch_holds_a_tree_of_fewer_nodes(box_scene):
    """75,777 triangles and a tree of 151,551 nodes: the scratch is sized for up to 2T = 151,554 nodes, whose sort has
    fewer tiles (of 2,048 keys) than that of 151,551 nodes (of 1,024).  The tree is regrouped as asked."""
    tris = soup(75777, 3)
    tris["material"] = 0
    sc = lumina.Scene(box_scene.camera, box_scene.sun, tris, box_scene.mat_albedo, box_scene.mat_emissive,
                      box_scene.points)
    nodes = heap_tree(tris, 75776)
    assert len(nodes) == 151551
    with lumina.Renderer(0) as r:
        r.set_render_tree("ploc")
        r.set_scene_bvh(sc, nodes)
        assert r.render_tree() == "ploc"
