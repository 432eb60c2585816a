"""After a pass of the device sort has given up (its error word is set), the kernels queued behind it touch no
row: they would read row ids that were never written.  The error word is set by the host here, before the
launch, over inputs that are whole; nothing is left to wait for."""
import ctypes as C

import numpy as np
import pytest

from minilake_b200 import abi

pytestmark = pytest.mark.gpu
N = 20_000  # three tiles of 8,192 rows
TILES = 3


class Col(C.Structure):
    _fields_ = [("dt", C.c_int32), ("kind", C.c_int32), ("src", C.c_int32), ("dict_len", C.c_uint32), ("data", C.c_void_p),
                ("off", C.c_void_p), ("valid", C.c_void_p), ("gid", C.c_void_p), ("dbytes", C.c_void_p), ("n", C.c_int64)]


class Word(C.Structure):
    _fields_ = [("col", Col), ("what", C.c_int32), ("chunk", C.c_int32), ("desc", C.c_int32), ("nulls_first", C.c_int32),
                ("rank", C.c_void_p)]


class Seg(C.Structure):
    _fields_ = [("word", C.c_int32), ("shift", C.c_int32), ("pos", C.c_int32), ("mask", C.c_uint32), ("sub", C.c_uint64)]


class Segs(C.Structure):
    _fields_ = [("n", C.c_int32), ("s", Seg * 32)]


def _launcher(name, *types):
    from minilake_b200.gpu import LIB
    f = getattr(LIB, name)
    f.argtypes = types
    return f


def _u32(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("gave_up", [False, True])
def test_kernels_behind_a_pass(gave_up):
    import torch
    P, I64, I32 = C.c_void_p, C.c_int64, C.c_int32
    keys_fn = _launcher("_ZN3mlg16launch_sort_keysEPKNS_8SortWordERKNS_8SortSegsEPKjlPjiS8_S7_P11CUstream_st",
                        P, C.POINTER(Segs), P, I64, P, I32, P, P, P)
    pass_fn = _launcher("_ZN3mlg17launch_radix_passEPKjS1_liS1_PmPjS3_S3_S3_P11CUstream_st",
                        P, P, I64, I32, P, P, P, P, P, P, P)
    runs_fn = _launcher("_ZN3mlg16launch_sort_runsEPKjPjPKNS_8SortWordEilP5uint2jS2_S1_P11CUstream_st",
                        P, P, P, I32, I64, P, C.c_uint32, P, P, P)
    dev = torch.device("cuda:0")
    r = np.random.default_rng(5)
    v = r.integers(0, 256, N)  # the key: one digit, the value above its lowest bit
    value = torch.from_numpy(v * 2 + r.integers(0, 2, N)).to(dev)
    col = Col(abi.INT64, 0, 0, 0, value.data_ptr(), None, None, None, None, N)
    word = torch.from_numpy(np.frombuffer(bytes(Word(col, 0, 0, 0, 0, None)), dtype=np.uint8).copy()).to(dev)
    segs = Segs(1)
    segs.s[0] = Seg(0, 1, 0, 0xFF, 1 << 63)
    i32 = dict(dtype=torch.int32, device=dev)
    rows_in = torch.arange(N, **i32)
    err = torch.full((1,), 1 if gave_up else 0, **i32)
    # the keys and their histogram
    keys = torch.full((N,), 7, **i32)
    hist = torch.zeros(256, **i32)
    keys_fn(word.data_ptr(), C.byref(segs), rows_in.data_ptr(), N, keys.data_ptr(), 1, hist.data_ptr(), err.data_ptr(), None)
    torch.cuda.synchronize()
    want_hist = np.bincount(v, minlength=256)
    assert np.array_equal(_u32(keys), np.full(N, 7) if gave_up else v)
    assert np.array_equal(_u32(hist), np.zeros(256) if gave_up else want_hist)
    # a pass over them
    keys = torch.from_numpy(v.astype(np.int32)).to(dev)
    start = torch.from_numpy(want_hist.astype(np.int32)).to(dev)
    status = torch.zeros(TILES * 256, dtype=torch.int64, device=dev)
    counter = torch.zeros(1, **i32)
    rows = torch.full((N,), 7, **i32)
    keys_out = torch.full((N,), 7, **i32)
    pass_fn(keys.data_ptr(), rows_in.data_ptr(), N, 0, start.data_ptr(), status.data_ptr(), counter.data_ptr(),
            keys_out.data_ptr(), rows.data_ptr(), err.data_ptr(), None)
    torch.cuda.synchronize()
    order = np.argsort(v, kind="stable")
    assert np.array_equal(_u32(rows), np.full(N, 7) if gave_up else order)
    assert np.array_equal(_u32(keys_out), np.full(N, 7) if gave_up else v[order])
    assert int(counter.item()) == TILES
    kind = status.cpu().numpy().view(np.uint64) >> np.uint64(62)
    assert np.all(kind == (3 if gave_up else 2))  # nothing to wait for: given up, or a prefix
    # pairs of equal keys, out of order by the value below the key
    few = np.repeat(np.arange(N // 2), 2)
    value2 = torch.from_numpy(few * 2 + np.tile([1, 0], N // 2)).to(dev)
    col2 = Col(abi.INT64, 0, 0, 0, value2.data_ptr(), None, None, None, None, N)
    word2 = torch.from_numpy(np.frombuffer(bytes(Word(col2, 0, 0, 0, 0, None)), dtype=np.uint8).copy()).to(dev)
    keys = torch.from_numpy(few.astype(np.int32)).to(dev)
    rows = torch.arange(N, **i32)
    cap = N // 2
    runs = torch.zeros(2 * cap, **i32)
    state = torch.zeros(2, **i32)
    runs_fn(keys.data_ptr(), rows.data_ptr(), word2.data_ptr(), 1, N, runs.data_ptr(), cap, state.data_ptr(), err.data_ptr(), None)
    torch.cuda.synchronize()
    swapped = np.arange(N).reshape(-1, 2)[:, ::-1].ravel()
    assert np.array_equal(_u32(rows), np.arange(N) if gave_up else swapped)
    assert _u32(state).tolist() == [0 if gave_up else cap, 0]
