"""The scan of counts about its kernels' bounds (a block's 4,096 counts, the 65,536 one launch takes): string
offsets of a column of that many strings are its sums, checked through the decode of a Parquet file against the
CPU restatement, and through a filter's compaction of that many rows' chunks."""
import numpy as np
import pytest

from test_gpu_parquet import _check_file, _write

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200 import gpu
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 8192, 65535, 65536, 65537, 131073])
def test_string_offsets(ctx, tmp_path, n):
    import pyarrow as pa
    r = np.random.default_rng(n)
    t = pa.table({"s": pa.array([f"{i:x}" * int(k) for i, k in enumerate(r.integers(0, 5, n))], pa.string())})
    path = str(tmp_path / "t.parquet")
    _write(path, t, row_group_size=n, use_dictionary=False, compression="NONE")
    _check_file(ctx, path)


@pytest.mark.parametrize("chunks", [1, 4096, 4097, 12289])
def test_compaction_of_many_chunks(ctx, chunks):
    import ctypes as C

    import torch
    from minilake_b200 import abi, gpu
    from minilake_b200.abi import BOOL, INT32, Col, Lit
    from minilake_b200.serving import DeviceTable
    n = chunks * 2048 - 5
    d = torch.randint(0, 100, (n,), dtype=torch.int32, device="cuda", generator=torch.Generator("cuda").manual_seed(chunks))
    t, out, k = DeviceTable([(INT32, d, None)]), torch.zeros(n, dtype=torch.int32, device="cuda"), C.c_int64()
    keep = abi.Keep()
    e = abi.encode_expr(Col(0) < Lit(37), BOOL, keep)
    arr, nc, rows = t.ml
    torch.cuda.synchronize()
    gpu._check(gpu.LIB.ml_gpu_filter(ctx.h, C.byref(e), arr, nc, rows, None, 0, abi.LOC_DEVICE, out.data_ptr(), C.byref(k)))
    want = torch.nonzero(d < 37).flatten().to(torch.int32)
    assert k.value == len(want) and torch.equal(out[:k.value], want)
