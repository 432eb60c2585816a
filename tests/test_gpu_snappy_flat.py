"""Snappy pages of few elements, which one block copies: literals of every alignment and length form,
stray copies (overlapping themselves, reading each other, reaching to the start), element counts and
spans about the path's limits, and streams it must leave to the passes that report them.  The same
bytes as pyarrow's decompressor, or a refusal where it refuses."""
import numpy as np
import pytest

import snappy_streams as ss

pytestmark = pytest.mark.gpu


def _build(parts, rng):
    """(data, stream) of parts: n > 0 a literal of n random bytes, (off, len) a copy."""
    out, elems = bytearray(), []
    for p in parts:
        if isinstance(p, tuple):
            for _ in range(p[1]):
                out.append(out[-p[0]])
            elems.append(ss.copy(*p))
        else:
            b = rng.integers(0, 256, p, dtype=np.uint8).tobytes()
            out += b
            elems.append(ss.literal(b))
    return bytes(out), b"".join(elems)


def _pad(parts):
    """Up to a whole number of 8-byte values."""
    n = sum(p[1] if isinstance(p, tuple) else p for p in parts)
    return parts + [8 - n % 8] if n % 8 else parts


CASES = {
    "one": [8],
    "lengths": [60, 61, 255, 256, 257, 65536, 65537, 7, 9],
    "odd": [1001, 1003, 1007, 1015, 1017, 2001],
    "overlap": [300, (1, 64), (3, 64), 700, (64, 64), (63, 61), 900],
    "chained": [500, (500, 64), (10, 60), (64, 64), 400, (1024, 64), 301],
    "far": [70_000, (69_999, 64), 70_000, (100_000, 33)],
    "at_64": [600] * 64,
    "at_65": [600] * 65,
    "sparse": [3000] + [(5, 4)] * 11,
    "dense": [256, 254, 250] + [10] * 200,
    "big": [(1 << 20) + 3],
    "tiny": [3, (1, 5), 6, (6, 7), (2, 64), 1, (80, 30), 2],
    "tiny_256": [8] + [(8, 8), 7] * 127 + [(3, 15)],
    "tiny_257": [8] + [(8, 8), 7] * 128,
    "tiny_4096": [4000, (4000, 64), 32],
    "above_4096": [4000, (4000, 64), 40],
}


def _decode(stream, data, tmp_path):
    import pyarrow as pa
    import pyarrow.parquet as pq
    from minilake_b200 import gpu, parquet
    path = str(tmp_path / "u.parquet")
    values = np.frombuffer(data, dtype=np.int64)
    schema = pa.schema([pa.field("v", pa.int64(), nullable=False)])
    pq.write_table(pa.table({"v": pa.array(values)}, schema=schema), path, compression="NONE", use_dictionary=False,
                   data_page_size=1 << 24, max_rows_per_page=1 << 20)
    chunk = ss.recompress_chunk(parquet.chunk_bytes(path, pq.ParquetFile(path).metadata.row_group(0).column(0)), lambda _: stream)
    ctx = gpu.Context(0)
    try:
        got = gpu.parquet_decode(ctx, chunk, parquet.PHYSICAL["INT64"], 0, parquet.CONV_INT64, 0, parquet.CODECS["SNAPPY"],
                                 len(values), 0)
        out = got.fetch()[0].values.copy()
        got.close()
        return out
    finally:
        ctx.close()


@pytest.mark.parametrize("name", CASES)
def test_few_elements(name, tmp_path):
    import pyarrow as pa
    data, body = _build(_pad(CASES[name]), np.random.default_rng(len(name)))
    stream = ss.varint(len(data)) + body
    assert pa.Codec("snappy").decompress(stream, len(data)).to_pybytes() == data
    assert np.array_equal(_decode(stream, data, tmp_path), np.frombuffer(data, dtype=np.int64))


@pytest.mark.parametrize("fault", ["short", "long", "offset", "zero", "length", "varint"])
def test_malformed_streams_are_refused(fault, tmp_path):
    from minilake_b200 import gpu
    data, body = _build([800, (300, 40), 760], np.random.default_rng(1))
    n = len(data)
    assert n % 8 == 0
    stream = ss.varint(n) + body
    if fault == "short":
        stream = stream[:-1]
    elif fault == "long":
        stream += ss.literal(b"x")
    elif fault == "offset":
        stream = ss.varint(n) + ss.literal(data[:800]) + ss.copy(801, 40) + ss.literal(data[840:])
    elif fault == "zero":
        stream = ss.varint(n) + ss.literal(data[:800]) + bytes([2 | (39 << 2), 0, 0]) + ss.literal(data[840:])
    elif fault == "length":
        stream = ss.varint(n + 8) + body
    else:
        stream = b"\xff\xff\xff\xff\xff\xff"
    with pytest.raises(gpu.MiniLakeError):
        _decode(stream, data, tmp_path)
