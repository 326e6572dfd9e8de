"""The radix sort at the sizes where its dispatch changes (one block up to 2048 and 8192 keys, then
tiles of 2048, 4096 and 8192 keys), against numpy's stable sort."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("bits", [1, 13, 64])
@pytest.mark.parametrize("n", [2, 33, 2047, 2048, 2049, 8191, 8192, 8193, 10240, 524288, 524289, 1 << 20,
                               (1 << 20) + 1, 3_000_001])
def test_sizes(ctx, n, bits):
    from xnyzip_b200 import _native as N
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64, endpoint=False) if bits < 64 else \
        rng.integers(0, np.iinfo(np.uint64).max, n, dtype=np.uint64)
    keys[n // 2:n // 2 + n // 8] = keys[0]  # a run of equal keys: stability
    order = np.argsort(keys, kind="stable")
    for payload in (False, True):
        k = torch.from_numpy(keys.view(np.int64).copy()).cuda()
        v = torch.arange(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        N.check(N.stage_sort(ctx.handle, C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()) if payload else None, n,
                             bits))
        assert np.array_equal(k.cpu().numpy().view(np.uint64), keys[order])
        if payload:
            assert np.array_equal(v.cpu().numpy(), order)
