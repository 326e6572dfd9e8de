"""Block streams with blocks that hold no units (which no encoder writes but the format allows), against
the oracle: the others keep their order and their units.  Also block counts that wrap modulo 2^64."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def streams_of(raw, count):
    """Head, [(meta, data)], tail of a -normal container."""
    params = struct.unpack_from("<Q", raw, 8)[0]
    at = 16 + 4 * params + 14
    head, out = raw[:at], []
    for _ in range(count):
        n, m = struct.unpack_from("<QQ", raw, at)
        at += 16
        out.append((raw[at:at + m], raw[at + m:at + m + n]))
        at += m + n
    return head, out, raw[at:]


def unpack(meta, data):
    n, width = struct.unpack("<I", meta[:4])[0], meta[4]
    v, bits = int.from_bytes(data, "little"), (1 << width) - 1
    mask, total, out = (1 << 64) - 1, 0, []
    for i in range(n):
        total = (total + ((v >> (i * width)) & bits)) & mask
        out.append(total)
    return out


def pack(values, width):
    mask, last, word = (1 << 64) - 1, 0, 0
    for i, x in enumerate(values):
        word |= ((x - last) & mask) << (i * width)
        last = x
    return struct.pack("<IB", len(values), width), word.to_bytes((len(values) * width + 7) // 8, "little")


def with_empty_blocks(raw, at):
    """The container with an empty block put before each block index in `at` (ids of their own)."""
    head, s, tail = streams_of(raw, 6)
    ids, counts = unpack(*s[0]), unpack(*s[1])
    for i in sorted(at, reverse=True):
        ids.insert(i, ids[min(i, len(ids) - 1)] + 7)
        counts.insert(i, 0)
    s[0], s[1] = pack(ids, 64), pack(counts, 64)
    return head + b"".join(struct.pack("<QQ", len(d), len(m)) + m + d for m, d in s) + tail


@pytest.mark.parametrize("n,extent", [(1, 10.0), (300, 900.0), (2048, 1e5), (5000, 1e5), (9000, 3000.0)])
def test_empty_blocks_are_skipped(ctx, oracle, n, extent):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, extent, (n, 3)).astype(np.float32)
    for hil in (0, 1):
        raw = oracle.compress(x, "cube", 0.8660254, hil, 0, 0, zstd=False)
        plain = oracle.decompress(raw, "cube", 0.8660254, 0, zstd=False)
        blocks = struct.unpack("<I", streams_of(raw, 6)[1][0][0][:4])[0]
        for at in ([0], [blocks], list(range(0, blocks, 3)), [blocks // 2] * 2100):
            made = with_empty_blocks(raw, at)
            want = oracle.decompress(made, "cube", 0.8660254, 0, zstd=False)
            assert want.tobytes() == plain.tobytes()
            got = ctx.decompress(made, 0, 0.8660254, False, False)
            assert np.asarray(got).tobytes() == want.tobytes()
