"""Units of the sorted keys against the oracle around the tile sizes (1024 keys below 2^19 points, 4096
from there on): duplicates that span tiles, every quad delta, both modes, -rle and -normal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1024, 1025, 2049, (1 << 19) - 1, 1 << 19, (1 << 19) + 1])
def test_units_around_the_tiles(ctx, oracle, n):
    rng = np.random.default_rng(n)
    for extent, copies in ((300.0, 1), (6.0, 40)):
        x = rng.uniform(0, extent, (-(-n // copies), 3)).astype(np.float32)
        x = np.repeat(x, copies, axis=0)[:n]
        for rle, th in ((0, 0), (1, 0), (1, 1024)):
            want = oracle.compress(x, "to", 0.2, n & 1, rle, th, zstd=False)
            assert ctx.compress(x, 1, 0.2, n & 1, rle, th, use_zstd=False) == want
