"""Snappy streams whose elements meet the edges of the device decode's units: its 8,192-byte stream
blocks (elements and headers across them, a literal spanning several, a stream ending at or just past
one), its 64 KB output fragments (full, one byte, none short of full) and the depth of its copy
resolution (a run of one byte, copies each reading the one before).  Every stream is checked with
pyarrow's decompressor first; the device decode has to give the same bytes."""
import numpy as np
import pytest

import snappy_streams as ss

BLOCK, FRAG = 8192, 65536


def _long_form(b: bytes, nb: int) -> bytes:
    """A literal with its length in nb bytes (more than it needs: the format allows it)."""
    return bytes([(59 + nb) << 2]) + (len(b) - 1).to_bytes(nb, "little") + b


def _copy4(off: int, ln: int) -> bytes:
    return bytes([3 | ((ln - 1) << 2)]) + off.to_bytes(4, "little")


def _elements(n: int, rng, shape: str):
    """(data, stream) of n output bytes in elements of the given shape, none crossing a fragment."""
    out, elems, size = bytearray(), [ss.varint(n)], len(ss.varint(n))
    while len(out) < n:
        at = len(out) % FRAG
        room = min(n - len(out), FRAG - at)
        if shape == "literals":
            k = min(room, int(rng.integers(1, 70)))
        elif shape == "edges":  # sized so that a header starts 1..5 bytes before a block's end
            k = min(room, max(1, BLOCK - size % BLOCK - int(rng.integers(1, 6)) - 3))
        elif shape == "spanning":
            k = min(room, int(rng.choice([3, 60, 61, 256, 20_000, 65_536])))
        else:
            k = min(room, int(rng.integers(1, 9)))
        copies = shape in ("mixed", "deep", "edges") and at > 0 and (shape != "mixed" or rng.random() < 0.7)
        if copies:
            k = min(room, int(rng.integers(1, 65)) if shape != "deep" else int(rng.integers(4, 9)))
            off = int(rng.integers(1, at + 1)) if shape == "mixed" else min(at, int(rng.integers(1, 9)))
            e = _copy4(off, k) if rng.random() < 0.2 else ss.copy(off, k)
            for _ in range(k):
                out.append(out[-off])
            if shape == "edges" and size % BLOCK < BLOCK - 300:  # then a literal up to the block's end
                elems.append(e)
                size += len(e)
                room = min(n - len(out), FRAG - len(out) % FRAG) if len(out) < n else 0
                if not room:
                    continue
                k = min(room, max(1, BLOCK - size % BLOCK - int(rng.integers(1, 6)) - 3))
                b = rng.integers(0, 256, k, dtype=np.uint8).tobytes()
                out += b
                e = ss.literal(b)
        else:
            b = rng.integers(0, 256, k, dtype=np.uint8).tobytes()
            out += b
            e = _long_form(b, int(rng.integers(2, 5))) if rng.random() < 0.2 and k <= 255 else ss.literal(b)
        elems.append(e)
        size += len(e)
    return bytes(out), b"".join(elems)


SIZES = [8, 8_184, 8_192, 16_384, 65_528, 65_536, 65_544, 3 * FRAG, 200_000]
CASES = [(s, n) for s in ("mixed", "deep", "literals", "edges", "spanning") for n in SIZES]


def _stream(shape, n):
    return _elements(n, np.random.default_rng(n * 7 + len(shape)), shape)


@pytest.mark.parametrize("shape,n", CASES)
def test_streams_are_valid(shape, n):
    import pyarrow as pa
    data, stream = _stream(shape, n)
    assert len(data) == n
    assert pa.Codec("snappy").decompress(stream, n).to_pybytes() == data


@pytest.mark.gpu
@pytest.mark.parametrize("shape,n", CASES)
def test_streams_decode_on_the_device(shape, n, tmp_path):
    import pyarrow as pa
    import pyarrow.parquet as pq
    from minilake_b200 import gpu, parquet
    data, stream = _stream(shape, n)
    path = str(tmp_path / "u.parquet")
    values = np.frombuffer(data, dtype=np.int64)
    schema = pa.schema([pa.field("v", pa.int64(), nullable=False)])
    pq.write_table(pa.table({"v": pa.array(values)}, schema=schema), path, compression="NONE", use_dictionary=False,
                   data_page_size=1 << 24, max_rows_per_page=1 << 20)
    pf = pq.ParquetFile(path)
    assert pf.schema.column(0).max_definition_level == 0

    def compress(payload):
        assert payload == data  # one page of the values as they are
        return stream
    chunk = ss.recompress_chunk(parquet.chunk_bytes(path, pf.metadata.row_group(0).column(0)), compress)
    ctx = gpu.Context(0)
    got = gpu.parquet_decode(ctx, chunk, parquet.PHYSICAL["INT64"], 0, parquet.CONV_INT64, 0, parquet.CODECS["SNAPPY"],
                             len(values), 0)
    assert np.array_equal(got.fetch()[0].values, values)
    got.close()
    ctx.close()
