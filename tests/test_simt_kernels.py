"""The library on the CPU (simt_host.py): its kernels with the warps of a block, and the lanes of a
warp, taking their turns in either order between barriers, against the oracle."""
import pytest

import simt_host

ORDERS = [0, 1, 2, 3]


@pytest.mark.parametrize("order", ORDERS)
def test_containers_in_either_order(oracle, order):
    """One-block and chained sorts, block and direct mode, both curves and containers."""
    simt_host.run(f"""
from oracle import Oracle
o = Oracle()
simt.simt_order({order})
ctx = X.Context(0)
for n in (40, 1013, 9000):
    x = np.random.default_rng(n).uniform(0, 30, (n, 3)).astype(np.float32)
    for q, name, hil, rle, thr in ((1, "to", 1, 1, 0), (0, "cube", 0, 0, 0), (0, "cube", 1, 0, 1024)):
        raw = ctx.compress(x, q, 0.05, hil, rle, thr, use_zstd=False)
        no_fault()
        assert raw == o.compress(x, name, 0.05, hil, rle, thr, zstd=False)
        got = ctx.decompress(raw, q, 0.05, rle, is_zstd=False)
        no_fault()
        assert got.tobytes() == o.decompress(raw, name, 0.05, rle, zstd=False).tobytes()
""")


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("n", [30_000, 60_000, 200_000])
def test_blocks_that_decode_again(oracle, order, n):
    """Runs of the codeword 11 of the code 0, 10, 11, some thousand long: a block that starts inside
    one reads from the wrong bit as consistently as from the right one, assumes a wrong entry, and
    decodes again once the block before it has told."""
    simt_host.run(f"""
from oracle import Oracle
from test_gpu_stream_decode import container
simt.simt_order({order})
sym = np.where(np.random.default_rng({n}).random({n}) < 1 / 3000, 1, 3)
raw = container(sym, {{1: 1, 2: 2, 3: 2}})
got = X.Context(0).decompress(raw, 0, 0.05, 0, is_zstd=False)
no_fault()
assert got.tobytes() == Oracle().decompress(raw, "cube", 0.05, 0, zstd=False).tobytes()
""")


@pytest.mark.parametrize("period", ["runs", "three bits"])
def test_giving_a_stream_up_is_cheap(oracle, period):
    """Streams that never fall in step (one run of the codeword 11 of the code 0, 10, 11; the codeword 110
    of a code with lengths 2 to 4) go to the decoder with entry tables.  The blocks that find it out stop
    after some rounds, and those that start later at once: barriers over all 24 and 36 blocks."""
    simt_host.run(f"""
from oracle import Oracle
from test_gpu_stream_decode import container
sym, lens = np.full(220_000, 3), {{1: 1, 2: 2, 3: 2}}
sym[0] = 1
if {period!r} == "three bits":
    sym, lens = np.full(220_000, 8), {{1: 3, 2: 2, 3: 3, 4: 3, 5: 3, 6: 4, 7: 4, 8: 3}}
    sym[0] = 2
raw = container(sym, lens)
ctx = X.Context(0)
simt.simt_clear()
got = ctx.decompress(raw, 0, 0.05, 0, is_zstd=False)
no_fault()
assert "decode_stream_kernel" in simt.simt_kernels().decode()
runs = simt.simt_kernels().decode().count("decode_sync_kernel")
assert simt.simt_barriers(b"decode_sync_kernel") <= 400 * runs, simt.simt_barriers(b"decode_sync_kernel")
assert got.tobytes() == Oracle().decompress(raw, "cube", 0.05, 0, zstd=False).tobytes()
""")


@pytest.mark.parametrize("order", ORDERS)
def test_zstd_frames_by_a_block(order):
    """The frame decoder as the device compiles it: 128 threads, the first warp walking the next
    sequences' states while the other three write the output; against libzstd."""
    simt_host.run(f"""
import test_zstd_host as T
simt.simt_order({order})
ctx = X.Context(0)
frame, data = T._zstd(), [d[:50_000] for d in T._data() if d]
for level in (1, 19):
    frames = [frame(d, level) for d in data]
    out = [device(bytes(len(d))) for d in data]
    sizes = ctx.zstd_decompress_device([device(f) for f in frames], [len(f) for f in frames], out, [len(d) for d in data])
    no_fault()
    for n, p, d in zip(sizes, out, data):
        assert n == len(d) and ctypes.string_at(p, n) == d
""")
