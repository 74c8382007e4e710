"""The radix sort (csrc/radix_sort.cu) by itself, against numpy's stable sort: every tile shape at the sizes where
it begins, ends and has a ragged last tile, and with a poll limit of zero, at which a tile takes every count that is
not there yet from the keys of the tile it waits for, as after a wait that ran out."""
import ctypes as C

import numpy as np
import pytest

from lumina import _ffi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Scratch(C.Structure):  # lg::RadixSortScratch
    _fields_ = [("keys_alt", C.c_void_p), ("vals_alt", C.c_void_p), ("hist", C.c_void_p), ("tickets", C.c_void_p),
                ("state", C.c_void_p), ("zero_bytes", C.c_size_t), ("capacity", C.c_size_t), ("poll_limit", C.c_int)]


def _sort(keys, bits, poll_limit=None, bound_for=None):
    """keys sorted over bits [0, bits) with their input positions, by lg::radix_sort_pairs."""
    lib = C.CDLL(str(_ffi.LIB_PATH))
    size = lib._ZN2lg24radix_sort_scratch_bytesEm
    size.restype, size.argtypes = C.c_size_t, [C.c_size_t]
    bind = lib._ZN2lg15radix_sort_bindEPvm
    bind.restype, bind.argtypes = Scratch, [C.c_void_p, C.c_size_t]
    sort = lib._ZN2lg16radix_sort_pairsEPjS0_miiRKNS_16RadixSortScratchEP11CUstream_stbb
    sort.restype = C.c_int
    sort.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.POINTER(Scratch), C.c_void_p, C.c_bool,
                     C.c_bool]
    n, room = len(keys), bound_for or len(keys)
    k = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    mem = torch.full((size(room) + 256,), 255, dtype=torch.uint8, device="cuda")  # nothing may rest on cleared memory
    s = bind(mem.data_ptr(), room)
    if poll_limit is not None:
        assert s.poll_limit > 1000
        s.poll_limit = poll_limit
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    rc = sort(k.data_ptr(), v.data_ptr(), n, 0, bits, C.byref(s), stream.cuda_stream, False, False)
    assert rc == 0
    stream.synchronize()
    return k.cpu().numpy().view(np.uint32), v.cpu().numpy()


def _check(n, bits, seed, **kw):
    rng = np.random.default_rng(seed)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    keys[n // 3:n // 2] = keys[0]  # a run of equal keys
    order = np.argsort(keys & np.uint32((1 << bits) - 1), kind="stable")
    k, v = _sort(keys, bits, **kw)
    assert (v == order).all() and (k == keys[order]).all()


# 1,024 keys a tile up to 148 tiles, then 2,048, 4,096 and 8,192
EDGES = [1, 2, 1023, 1024, 1025, 20500, 148 * 1024, 148 * 1024 + 1, 200001, 148 * 2048, 148 * 2048 + 1, 400001,
         148 * 4096, 148 * 4096 + 1, 148 * 8192 + 5]


@pytest.mark.parametrize("n", EDGES)
def test_tile_shapes(n):
    _check(n, 30, n)


@pytest.mark.parametrize("n", [2, 1025, 20500, 148 * 1024, 200001, 400001, 700001])
@pytest.mark.parametrize("bits", [8, 30, 32])
def test_right_without_waiting(n, bits):
    _check(n, bits, n + bits, poll_limit=0)


@pytest.mark.parametrize("n,room", [(148 * 1024, 148 * 1024 + 1), (20500, 400001), (148 * 2048, 148 * 4096)])
def test_fewer_pairs_than_bound_for(n, room):
    _check(n, 30, n, bound_for=room)
