"""The ordered compaction of filters and join probes at the edges of its units (a 32-row word, a warp's
1,024 rows, a block's 2,048 and 8,192): selections and pairs against numpy, exactly, with none, some and
all rows kept, with an input selection, over a dense and a hashed join index, NULL keys, and results written
straight into device buffers (which must be left alone past the result)."""
import ctypes as C

import numpy as np
import pytest

from minilake_b200 import abi
from minilake_b200.abi import INT32, INT64, Col, Lit
from minilake_b200.columns import fixed

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 1023, 1024, 1025, 2047, 2048, 2049, 8191, 8192, 8193, 100_003]


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200.gpu import Context
    ctx = Context(0)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("keep", [0.0, 0.03, 0.9, 1.0])
def test_selections(ctx, n, keep):
    import torch
    from minilake_b200 import gpu
    r = np.random.default_rng(n)
    v = r.permutation(n).astype(np.int32)
    cut = int(round(keep * n))
    op = gpu.FilterOperator(ctx, Col(0) < Lit(cut))
    want = np.nonzero(v < cut)[0]
    batch = ctx.upload([fixed(INT32, v)])
    assert np.array_equal(op.execute(batch), want)
    sel = np.sort(r.choice(n, max(1, n // 2), replace=False)).astype(np.uint32)
    assert np.array_equal(op.execute(batch, sel), sel[v[sel] < cut])
    keepalive = abi.Keep()
    e = abi.encode_expr(Col(0) < Lit(cut), abi.BOOL, keepalive)
    arr, nc = batch.ml_columns()
    out, k = torch.full((n + 64,), -7, dtype=torch.int32, device="cuda"), C.c_int64()
    gpu._check(gpu.LIB.ml_gpu_filter(ctx.h, C.byref(e), arr, nc, n, None, 0, abi.LOC_DEVICE, out.data_ptr(), C.byref(k)))
    got = out.cpu().numpy()
    assert k.value == len(want) and np.array_equal(got[:k.value], want) and (got[k.value:] == -7).all()
    # in place: the input selection's own buffer receives the result
    buf = torch.from_numpy(sel.astype(np.int32)).cuda()
    gpu._check(gpu.LIB.ml_gpu_filter(ctx.h, C.byref(e), arr, nc, n, buf.data_ptr(), len(sel), abi.LOC_DEVICE, buf.data_ptr(), C.byref(k)))
    assert np.array_equal(buf.cpu().numpy()[:k.value], sel[v[sel] < cut])


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("spread", [1, 1 << 33])
def test_pairs(ctx, n, spread):
    import torch
    from minilake_b200 import gpu
    from minilake_b200.engine import GpuEngine
    r = np.random.default_rng(n)
    m = max(1, n // 3)
    build = r.permutation(m).astype(np.int64) * spread
    row = r.integers(0, 2 * m, n) * spread
    ok = r.random(n) > 0.1
    join = GpuEngine(ctx).join_build([ctx.upload([fixed(INT64, build)])], [INT64], [(Col(0), INT64)])
    at = np.full(2 * m, -1)
    at[build // spread] = np.arange(m)
    match = np.where(ok, at[row // spread], -1)
    want = np.nonzero(match >= 0)[0]
    batch = ctx.upload([fixed(INT64, row, ok)])
    probe = gpu.HashJoinProbe(ctx, join.handle, [(Col(0), INT64)])
    p, b = probe.execute(batch)
    assert np.array_equal(p, want) and np.array_equal(b, match[want])
    sel = np.sort(r.choice(n, max(1, n // 2), replace=False)).astype(np.uint32)
    p, b = probe.execute(batch, sel)
    assert np.array_equal(p, sel[match[sel] >= 0]) and np.array_equal(b, match[p])
    keepalive = abi.Keep()
    e, ne = abi.encode_exprs([(Col(0), INT64)], keepalive)
    arr, nc = batch.ml_columns()
    outs, k = [torch.full((n + 64,), -7, dtype=torch.int32, device="cuda") for _ in range(2)], C.c_int64()
    gpu._check(gpu.LIB.ml_gpu_join_probe(ctx.h, join.handle, e, ne, arr, nc, n, None, 0, abi.LOC_DEVICE, outs[0].data_ptr(),
                                         outs[1].data_ptr(), n, C.byref(k)))
    for out, ref in zip(outs, (want, match[want])):
        got = out.cpu().numpy()
        assert k.value == len(ref) and np.array_equal(got[:k.value], ref) and (got[k.value:] == -7).all()
