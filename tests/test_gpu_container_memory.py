"""decompress_device on containers in host memory that a device copy can read: copied, not read in place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [50, 3000, 60_000])
def test_pinned_container(ctx, oracle, n):
    from xnyzip_b200 import verify as V
    x = np.random.default_rng(n).uniform(0, 60, (n, 3)).astype(np.float32)
    raw = oracle.compress(x, "to", 0.05, 1, 1, 0, zstd=False)
    host = torch.frombuffer(bytearray(raw), dtype=torch.uint8).pin_memory()
    p, k = ctx.decompress_device(host.data_ptr(), len(raw), 1, 0.05, 1)
    got = V.device_view(p, (k, 3), "<f4", torch.device("cuda:0")).cpu().numpy()
    assert got.tobytes() == oracle.decompress(raw, "to", 0.05, 1, zstd=False).tobytes()
