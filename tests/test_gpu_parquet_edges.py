"""Parquet decode at the edges of its kernels: rows about a block's slice (512) and a tile (8,192),
pages that end inside a validity word, streams longer than the walk's window (8 KB) with runs of
both kinds, string dictionaries about the one-block bound (1,024 entries, 64 KB), and dictionaries
whose strings are too many for an encoded column.  Values, validity, dictionaries and codes are
compared with the CPU restatement bit for bit (tests/test_gpu_parquet.py)."""
import numpy as np
import pytest

from test_gpu_parquet import _check_file, _write

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from minilake_b200 import gpu
    return gpu.Context(0)


@pytest.mark.parametrize("version", ["1.0", "2.0"])
@pytest.mark.parametrize("rows,page", [(1, 20000), (31, 7), (511, 33), (512, 512), (513, 500), (8191, 20000), (8192, 8192),
                                       (8193, 1000), (70001, 20000)])
def test_rows_about_slices_tiles_and_pages(ctx, tmp_path, rows, page, version):
    import pyarrow as pa
    rng = np.random.default_rng(rows)
    null = rng.random(rows) < 0.3
    null[: rows // 2] = np.repeat(rng.random(rows // 2 // 40 + 1) < 0.5, 40)[: rows // 2]  # long runs, then mixed
    words = ["", "a", "bc", "def"]
    runs = np.repeat(rng.integers(0, 300, rows // 9 + 1), 9)[:rows]  # RLE and bit-packed runs of indices
    t = pa.table({
        "i32": pa.array(rng.integers(-2**31, 2**31 - 1, rows, dtype=np.int32), mask=null),
        "run": pa.array(runs.astype(np.int64), mask=null),
        "few": pa.array(np.array(words, dtype=object)[rng.integers(0, 4, rows)], mask=null, type=pa.string()),
        "b": pa.array(rng.random(rows) < 0.5, mask=null),
        "f64": pa.array(rng.normal(size=rows)),
        "none": pa.array([None] * rows, pa.string()),
    })
    for kw in ({}, {"use_dictionary": False}):
        path = str(tmp_path / f"t{len(kw)}.parquet")
        _write(path, t, row_group_size=rows, data_page_version=version, max_rows_per_page=page, **kw)
        _check_file(ctx, path)


@pytest.mark.parametrize("entries,length", [(1, 3), (1022, 5), (1023, 5), (1024, 5), (1025, 5), (40, 1630), (40, 1640)])
@pytest.mark.parametrize("rows", [2000, 30011])
def test_string_dictionaries_about_the_one_block_bound(ctx, tmp_path, entries, length, rows):
    """With 2,000 rows most of these have more strings than an encoded column may (rows / 8)."""
    import pyarrow as pa
    rng = np.random.default_rng(entries + rows)
    words = np.array([(f"{i:x}" + "-" * length)[:length] if i else "" for i in range(entries)], dtype=object)
    pick = rng.permutation(np.concatenate([np.arange(entries), rng.integers(0, entries, rows - entries)]))
    for mask in (None, rng.random(rows) < 0.1):
        t = pa.table({"s": pa.array(words[pick], mask=mask, type=pa.string())})
        path = str(tmp_path / "t.parquet")
        _write(path, t, row_group_size=rows, max_rows_per_page=7000, compression="SNAPPY")
        _check_file(ctx, path)


def test_wide_indices_and_long_strings_cross_the_window(ctx, tmp_path):
    import pyarrow as pa
    rng = np.random.default_rng(5)
    rows = 60000
    t = pa.table({
        "wide": pa.array(rng.permutation(rows).astype(np.int64)),  # 16-bit indices: several windows a page
        "long": pa.array(["s" * int(n) + str(i) for i, n in enumerate(rng.integers(0, 300, rows))], pa.string()),
        "huge": pa.array([("h" * 9000 + str(i)) if i % 6000 == 0 else "x" for i in range(rows)], pa.string()),
    })
    for kw in ({"dictionary_pagesize_limit": 64 << 20}, {"use_dictionary": False}):
        path = str(tmp_path / f"t{len(kw)}{'d' if 'use_dictionary' in kw else ''}.parquet")
        _write(path, t, row_group_size=rows, compression="NONE", **kw)
        _check_file(ctx, path)
