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


def decode_at(ctx, raw, off, q, l2, rle):
    """Points of the container from an exactly sized device buffer, `off` bytes into it."""
    from xnyzip_b200 import verify as V
    buf = torch.zeros(off + len(raw), dtype=torch.uint8, device="cuda")
    buf[off:] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()
    torch.cuda.synchronize()
    p, n = ctx.decompress_device(buf.data_ptr() + off, len(raw), q, l2, rle)
    return V.device_view(p, (n, 3), "<f4", buf.device).cpu().numpy()


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("n,threshold", [(40, 0), (3000, 0), (3000, 1024), (60_000, 0)])
def test_containers_in_place_at_any_byte(ctx, oracle, n, threshold, off):
    """Small containers come to the host whole, large ones through the header kernel; those off a
    4-byte boundary are copied first."""
    x = np.random.default_rng(n).uniform(0, 30, (n, 3)).astype(np.float32)
    for rle in (0, 1):
        raw = oracle.compress(x, "to", 0.05, 1, rle, threshold, zstd=False)
        want = oracle.decompress(raw, "to", 0.05, rle, zstd=False)
        assert decode_at(ctx, raw, off, 1, 0.05, rle).tobytes() == want.tobytes()


@pytest.mark.parametrize("repeats", [400, 3000])
def test_meta_beyond_the_header_kernels_room(ctx, oracle, repeats):
    """A symbol table that lists its entries many times over (the last one counts): up to 78 KB."""
    import struct
    from test_gpu_stream_decode import canonical, container
    lens = {1: 1, 2: 2, 3: 2}
    sym = np.random.default_rng(5).integers(1, 4, 30_000)
    raw = container(sym, lens)
    table = canonical(lens)
    entry = b"".join(struct.pack(">QBI", s, ln, b) for s, (b, ln) in table.items())
    meta, many = struct.pack(">I", 3) + entry, struct.pack(">I", 3 * repeats) + entry * repeats
    data = struct.unpack_from("<Q", raw, 46)[0]
    big = raw[:46] + struct.pack("<QQ", data, len(many)) + many + raw[62 + len(meta):]
    want = oracle.decompress(raw, "cube", 0.05, 0, zstd=False)
    assert decode_at(ctx, big, 0, 0, 0.05, 0).tobytes() == want.tobytes()


def test_damaged_lengths_fail_cleanly(ctx, oracle, xnyz):
    x = np.random.default_rng(2).uniform(0, 100, (30_000, 3)).astype(np.float32)
    raw = oracle.compress(x, "to", 0.05, 1, 1, 0, zstd=False)
    for cut in (0, 7, 30, 63, 70, len(raw) // 2, len(raw) - 13, len(raw) - 1):
        with pytest.raises(xnyz.XnyzError):
            decode_at(ctx, raw[:cut] or b"\0", 0, 1, 0.05, 1)
    bad = bytearray(raw)
    bad[30 + 5] = 0xFF  # the first stream's length
    with pytest.raises(xnyz.XnyzError):
        decode_at(ctx, bytes(bad), 0, 1, 0.05, 1)
    assert decode_at(ctx, raw, 0, 1, 0.05, 1).shape == x.shape
