"""Entropy-coded streams with long runs of one codeword, which read as consistently from a wrong bit as
from the right one, against the oracle's sequential decoder."""
import numpy as np
import pytest

from test_gpu_stream_decode import check, container

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean_run", [900, 3000, 20_000])
@pytest.mark.parametrize("n", [30_000, 200_000, 3_000_000])
def test_blocks_that_decode_again(ctx, oracle, n, mean_run):
    """Codes 0, 10, 11 with runs of 11 in between: the blocks inside a run assume a wrong entry."""
    sym = np.where(np.random.default_rng(n).random(n) < 1 / mean_run, 1, 3)
    raw = container(sym, {1: 1, 2: 2, 3: 2})
    for _ in range(3):
        check(ctx, oracle, raw)
