"""zstd frames decoded on the GPU, by what their sequences are like: matches that overlap themselves
(periods from 1 byte), matches that repeat other matches of the same batch, sequences longer than a
chunk of output (2048 bytes), sequence counts around a batch (64), raw and one-stream literals, many
frames at once."""
import numpy as np
import pytest

from test_gpu_zstd import _gpu_decode, _libzstd, _zstd

pytestmark = pytest.mark.gpu


def periods(rng):
    return b"".join(rng.integers(0, 256, p, dtype=np.uint8).tobytes() * (int(rng.integers(3, 4000)) // p + 2)
                    for p in (1, 2, 3, 5, 7, 8, 9, 16, 31, 64, 300))


def words(rng, count):
    w = [rng.integers(97, 123, int(rng.integers(3, 9)), dtype=np.uint8).tobytes() for _ in range(60)]
    return b" ".join(w[int(i)] for i in rng.integers(0, 60, count))


def pieces(rng, count):
    """`count` copies of pieces of a random block, each behind a few fresh bytes: about one sequence each."""
    base = rng.integers(0, 256, 5000, dtype=np.uint8).tobytes()
    out = [base]
    for _ in range(count):
        at, n = int(rng.integers(0, 4900)), int(rng.integers(8, 60))
        out += [rng.integers(0, 256, int(rng.integers(1, 5)), dtype=np.uint8).tobytes(), base[at:at + n]]
    return b"".join(out)


@pytest.mark.parametrize("level", [1, 3, 19])
def test_sequences(ctx, level):
    z, rng = _libzstd(), np.random.default_rng(level)
    plains = [periods(rng), periods(rng)[::-1], words(rng, 20), words(rng, 300), words(rng, 30000),
              bytes(5000) + b"x" + bytes(3000), b"ab" * 40, rng.integers(0, 256, 3000, dtype=np.uint8).tobytes() * 3]
    plains += [pieces(rng, k) for k in (1, 62, 63, 64, 65, 127, 128, 129, 1000)]
    frames = [_zstd(z, p, level) for p in plains]
    lens, outs, _, _ = _gpu_decode(ctx, frames, [len(p) for p in plains])
    assert [int(n) for n in lens] == [len(p) for p in plains]
    assert outs == plains


def test_many_frames(ctx):
    z, rng = _libzstd(), np.random.default_rng(9)
    plains = [words(rng, int(rng.integers(1, 2000))) for _ in range(1000)]
    frames = [_zstd(z, p, 3) for p in plains]
    assert _gpu_decode(ctx, frames, [len(p) for p in plains])[1] == plains
