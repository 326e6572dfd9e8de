"""The entropy decoders on hand-made direct-mode containers (any code, any size), against the
oracle's sequential decoder: sizes around the blocks of the self-synchronising decoder, codes
whose wrong offsets never fall in step (the entry-table decoder takes those), codes longer than
the primary table, and Golomb-Rice values beyond 32 bits."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def canonical(lens):
    """{symbol: (bits, length)} of a canonical prefix code."""
    code, out, prev = 0, {}, 0
    for ln, s in sorted((ln, s) for s, ln in lens.items()):
        code <<= ln - prev
        out[s] = (code, ln)
        code += 1
        prev = ln
    assert code <= 1 << prev
    return out


def container(symbols, lens, hilbert=0):
    """Direct-mode -normal container: SFC deltas symbol - 1, no patches."""
    table = canonical(lens)
    bits = "".join(format(table[s][0], f"0{table[s][1]}b") for s in symbols.tolist())
    data = np.packbits(np.frombuffer(bits.encode(), np.uint8) - 48).tobytes()
    meta = struct.pack(">I", len(table)) + b"".join(struct.pack(">QBI", s, ln, b) for s, (b, ln) in table.items())
    head = struct.pack("<QQiiiBB", len(symbols), 0, 1 << 19, 1 << 19, 1 << 19, hilbert, 1)
    return head + struct.pack("<QQ", 0, 0) + struct.pack("<QQ", len(data), len(meta)) + meta + data + \
        struct.pack("<fff", 1.0, -2.0, 0.5)


def check(ctx, oracle, raw):
    got = ctx.decompress(raw, 0, 0.05, 0, is_zstd=False)
    assert got.tobytes() == oracle.decompress(raw, "cube", 0.05, 0, zstd=False).tobytes()


SKEWED = {1: 1, 2: 3, 3: 3, 4: 4, 5: 5, 6: 6, 7: 6}
FLAT = {s: (4 if s < 6 else 5 if s < 10 else 6) for s in range(1, 30)}


# bits per subsequence x threads of a block: 160 and 288 bits x 128 (the smallest), the block's own
# subsequences 116 (12 are decoded ahead); sizes in codewords of `code` on either side of them
@pytest.mark.parametrize("code", ["skewed", "flat"])
@pytest.mark.parametrize("n", [2, 31, 159, 160, 161, 4000, 10500, 20480, 20600, 61000, 400_003])
def test_sizes_around_the_blocks(ctx, oracle, code, n):
    lens = SKEWED if code == "skewed" else FLAT
    rng = np.random.default_rng(n)
    p = np.array([2.0 ** -ln for ln in lens.values()])
    sym = rng.choice(list(lens), n, p=p / p.sum())
    sym[:2] = list(lens)[:2]
    check(ctx, oracle, container(sym, lens))


@pytest.mark.parametrize("n", [500, 30_000, 300_000])
def test_code_that_never_falls_in_step(ctx, oracle, n):
    """Almost only the codeword 110 of a code with lengths 1..4: a wrong offset reads 1 0 1 1 0 ..,
    other codewords with the same period."""
    lens = {1: 3, 2: 2, 3: 3, 4: 3, 5: 3, 6: 4, 7: 4, 8: 3}
    sym = np.full(n, 8)
    sym[0] = 2
    check(ctx, oracle, container(sym, lens))


@pytest.mark.parametrize("n", [300, 50_000])
def test_lengths_with_a_common_divisor(ctx, oracle, n):
    lens = {1: 2, 2: 2, 3: 2, 4: 4, 5: 4, 6: 4, 7: 4}
    sym = np.random.default_rng(n).integers(1, 8, n)
    check(ctx, oracle, container(sym, lens))


@pytest.mark.parametrize("n", [40, 3000, 90_000])
def test_codes_longer_than_the_tables(ctx, oracle, n):
    lens = {s: s for s in range(1, 25)} | {25: 24}
    rng = np.random.default_rng(n)
    sym = np.where(rng.random(n) < 0.2, rng.integers(9, 26, n), np.minimum(rng.geometric(0.5, n), 25))
    check(ctx, oracle, container(sym, lens))


@pytest.mark.parametrize("n", [3, 50, 700, 20_000])
@pytest.mark.parametrize("extent", [40.0, 3000.0, 60000.0])
def test_golomb_rice_values_beyond_32_bits(ctx, oracle, n, extent):
    """Direct mode over up to 2^20 cells per axis: deltas of up to 60 bits, Golomb-Rice
    parameters from 0 to above 32."""
    x = np.random.default_rng(n).uniform(0, extent, (n, 3)).astype(np.float32)
    for hil in (0, 1):
        raw = ctx.compress(x, 0, 0.05, hil, 0, 1 << 20, use_zstd=False)
        assert raw == oracle.compress(x, "cube", 0.05, hil, 0, 1 << 20, zstd=False)
        check(ctx, oracle, raw)
