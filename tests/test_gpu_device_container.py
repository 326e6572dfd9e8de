"""The device container (xnyz_compress_device), whose block streams are packed straight into place,
against the oracle's: block counts around the packing tile (2048), id widths from a few bits to
over 32, count deltas that wrap (64 bits) or need one bit, every byte alignment of the second stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

QN = {0: "cube", 1: "to", 2: "adaptive"}


def device_container(ctx, x, q, l2, hil, rle):
    from xnyzip_b200 import verify as V
    d = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    p, n = ctx.compress_device(d.data_ptr(), x.shape[0], q, l2, hil, rle, 0)
    return V.device_view(p, (n,), "|u1", d.device).cpu().numpy().tobytes()


@pytest.mark.parametrize("extent", [150.0, 3000.0, 1e5, 5e5])
@pytest.mark.parametrize("n", [1, 2, 5, 33, 2046, 2047, 2048, 2049, 2050, 4096, 4097, 9001])
def test_block_streams_in_place(ctx, oracle, n, extent):
    rng = np.random.default_rng(n + int(extent))
    x = rng.uniform(0, extent, (n, 3)).astype(np.float32)
    for q, l2, rle in ((0, 0.8660254, 1), (1, 0.5, 0), (2, 0.5, 1)):
        want = oracle.compress(x, QN[q], l2, 1, rle, 0, zstd=False)
        assert device_container(ctx, x, q, l2, 1, rle) == want


@pytest.mark.parametrize("n", [700, 2047, 2048, 2049, 2055])
def test_equal_counts_need_one_bit(ctx, oracle, n):
    """One point per block, the blocks a constant step apart: both streams narrower than a byte."""
    x = np.zeros((n, 3), np.float32)
    x[:, 0] = np.arange(n) * 128.0 + 5
    want = oracle.compress(x, "cube", 0.8660254, 0, 1, 0, zstd=False)
    assert device_container(ctx, x, 0, 0.8660254, 0, 1) == want
