"""A context after a call that failed: the next calls' results are the oracle's."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_container_with_a_short_count_stream(ctx, oracle, xnyz):
    """The count stream of a large container is cut: the host finds that the code cannot fit and returns
    at once, the container's memory is overwritten, and the context goes on."""
    rng = np.random.default_rng(3)
    x = rng.uniform(0, 4000, (400_000, 3)).astype(np.float32)
    x = np.concatenate([x, x[:200_000]])  # counts 1 and 2: one bit each
    raw = oracle.compress(x, "to", 0.05, 1, 1, 0, zstd=False)
    at = 16 + 14
    for _ in range(6):
        dl, ml = struct.unpack_from("<QQ", raw, at)
        at += 16 + ml + dl
    dl, ml = struct.unpack_from("<QQ", raw, at)
    bad = raw[:at] + struct.pack("<QQ", dl // 2, ml) + raw[at + 16:at + 16 + ml + dl // 2] + raw[-12:]
    y = rng.uniform(0, 300, (50_000, 3)).astype(np.float32)
    want = oracle.compress(y, "to", 0.05, 1, 1, 0, zstd=False)
    points = oracle.decompress(want, "to", 0.05, 1, zstd=False)
    for _ in range(5):
        d = torch.frombuffer(bytearray(bad), dtype=torch.uint8).cuda()
        torch.cuda.synchronize()
        with pytest.raises(xnyz.XnyzError):
            ctx.decompress_device(d.data_ptr(), len(bad), 1, 0.05, 1)
        d.fill_(255)
        assert ctx.compress(y, 1, 0.05, 1, 1, 0, use_zstd=False) == want
        assert ctx.decompress(want, 1, 0.05, 1, is_zstd=False).tobytes() == points.tobytes()
