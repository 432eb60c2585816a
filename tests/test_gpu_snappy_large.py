"""Snappy pages larger than the device decode takes at once (32 MB of stream): their parts' edges fall anywhere
in elements and fragments, long literals span them, and the memory that the decode's tables take does not grow
with the page.  The device decode has to give the bytes the stream was made from."""
import numpy as np
import pytest

import snappy_streams as ss
from test_gpu_snappy_blocks import FRAG, _elements

MB = 1 << 20


def _stream(shape, mb):
    """At least `mb` MB of stream: pieces of whole fragments, whose copies stay within their fragment."""
    pieces = []
    for seed in range(3):
        data, stream = _elements(5 * FRAG, np.random.default_rng(seed), shape)
        head = len(ss.varint(len(data)))
        pieces.append((data, stream[head:]))
    out, elems, size, k = [], [], 0, 0
    while size < mb * MB:
        data, body = pieces[k % 3]
        out.append(data)
        elems.append(body)
        size += len(body)
        k += 1
    data = b"".join(out)
    return data, ss.varint(len(data)) + b"".join(elems)


@pytest.mark.parametrize("shape", ["mixed", "literals"])
def test_streams_are_valid(shape):
    import pyarrow as pa
    data, stream = _stream(shape, 2)
    assert pa.Codec("snappy").decompress(stream, len(data)).to_pybytes() == data


@pytest.mark.gpu
@pytest.mark.parametrize("shape,mb", [("mixed", 33), ("literals", 33), ("edges", 70), ("spanning", 96)])
def test_pages_in_parts(shape, mb, tmp_path):
    import pyarrow as pa
    import pyarrow.parquet as pq
    import torch
    from minilake_b200 import gpu, parquet
    data, stream = _stream(shape, mb)
    assert len(stream) > 32 * MB
    values = np.frombuffer(data, dtype=np.int64)
    path = str(tmp_path / "u.parquet")
    schema = pa.schema([pa.field("v", pa.int64(), nullable=False)])
    pq.write_table(pa.table({"v": pa.array(values)}, schema=schema), path, compression="NONE", use_dictionary=False,
                   data_page_size=1 << 30, max_rows_per_page=1 << 30, row_group_size=1 << 30, write_batch_size=1 << 26)
    meta = pq.ParquetFile(path).metadata.row_group(0).column(0)

    def compress(payload):
        assert payload == data  # one page of the values as they are
        return stream
    chunk = ss.recompress_chunk(parquet.chunk_bytes(path, meta), compress)
    ctx = gpu.Context(0)

    def decode(chunk, rows):
        out = gpu.parquet_decode(ctx, chunk, parquet.PHYSICAL["INT64"], 0, parquet.CONV_INT64, 0, parquet.CODECS["SNAPPY"], rows, 0)
        got = out.fetch()[0].values
        out.close()
        return got
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        assert np.array_equal(decode(chunk, len(values)), values)
    # the run tables take 32 bytes a row, the page, its chunk and the column some 8 each; the Snappy tables 512 MB
    assert free - torch.cuda.mem_get_info()[0] < 64 * len(values) + (640 << 20)
    ctx.close()
