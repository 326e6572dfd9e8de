"""Huffman streams whose codewords all have one length (1 to 8 bits for the symbols, 1 to 11 for the
-rle counts), decoded 16 symbols per thread, against the oracle: stream lengths around 16 symbols and a
block's share, every bit alignment of the second stream, a chunk that is no codeword."""
import struct

import numpy as np
import pytest

from test_gpu_stream_decode import canonical

pytestmark = pytest.mark.gpu


def stream(values, table, entry):
    bits = "".join(format(table[s][0], f"0{table[s][1]}b") for s in values.tolist())
    data = np.packbits(np.frombuffer(bits.encode(), np.uint8) - 48).tobytes()
    meta = struct.pack(">I", len(table)) + b"".join(entry(s) + struct.pack(">BI", ln, b) for s, (b, ln) in table.items())
    return struct.pack("<QQ", len(data), len(meta)) + meta + data


def container(symbols, lens, counts=None, count_lens=None):
    """Direct-mode container without patches, -rle with counts."""
    out = struct.pack("<QQiiiBB", len(symbols), 0, 1 << 19, 1 << 19, 1 << 19, 0, 1) + struct.pack("<QQ", 0, 0)
    out += stream(symbols, canonical(lens), lambda s: struct.pack(">Q", s))
    if counts is not None:
        out += stream(counts, canonical(count_lens), lambda s: struct.pack("<i", s))
    return out + struct.pack("<fff", 1.0, -2.0, 0.5)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 4095, 4096, 4097, 20_000])
def test_one_length(ctx, oracle, n):
    rng = np.random.default_rng(n)
    for length in range(1, 9):
        lens = {s: length for s in range(1, min(1 << length, 255) + 1)}
        raw = container(rng.integers(1, len(lens) + 1, n), lens)
        want = oracle.decompress(raw, "cube", 0.05, 0, zstd=False)
        assert ctx.decompress(raw, 0, 0.05, False, False).tobytes() == want.tobytes()
    for length in range(1, 12):
        lens, count_lens = {1: 1, 2: 1}, {s: length for s in range(1, (1 << length) + 1)}
        raw = container(rng.integers(1, 3, n), lens, rng.integers(1, min(len(count_lens), 40) + 1, n), count_lens)
        want = oracle.decompress(raw, "cube", 0.05, 1, zstd=False)
        assert ctx.decompress(raw, 0, 0.05, True, False).tobytes() == want.tobytes()


def test_a_chunk_that_is_no_codeword(ctx, xnyz):
    lens = {s: 3 for s in range(1, 8)}  # 111 is none
    raw = bytearray(container(np.ones(100, np.int64), lens))
    raw[-12 - 20] |= 0xff
    with pytest.raises(xnyz.XnyzError):
        ctx.decompress(bytes(raw), 0, 0.05, False, False)
    good = container(np.ones(100, np.int64), lens)
    assert len(ctx.decompress(good, 0, 0.05, False, False)) == 100
