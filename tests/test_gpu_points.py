"""Bounding box, quantization and keys against the oracle around the size (2^18 points) from which a thread
takes four points at a time, with the points on and off a 16-byte boundary: values on the lattice's
edges, zeros of both signs, coordinates near the float range's lower end, extents beyond 2^24 steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

QN = {0: "cube", 1: "to", 2: "adaptive"}
V = 1 << 18


def container(ctx, x, off, q, l2, hil, rle, th):
    """The device container of points that start `off` floats into an allocation."""
    from xnyzip_b200 import verify
    buf = torch.zeros(off + x.size, dtype=torch.float32, device="cuda")
    buf[off:] = torch.from_numpy(x.reshape(-1)).cuda()
    torch.cuda.synchronize()
    p, n = ctx.compress_device(buf.data_ptr() + 4 * off, x.shape[0], q, l2, hil, rle, th)
    return verify.device_view(p, (n,), "|u1", buf.device).cpu().numpy().tobytes()


def points(kind, n, rng):
    if kind == "edges":  # multiples of half a step, some moved by one unit in the last place
        step = np.float32(2.0 * 0.05 / np.sqrt(5.0))
        x = (rng.integers(0, 4000, (n, 3)) * (step / 2)).astype(np.float32)
        return np.where(rng.random((n, 3)) < 0.5, x, np.nextafter(x, np.float32(1e9)))
    if kind == "tiny":  # below 2^-60, zeros of both signs
        x = rng.uniform(0, 40, (n, 3)).astype(np.float32)
        m = rng.random((n, 3))
        x[m < 0.3] = np.float32(1e-30)
        x[m < 0.2] = np.float32(0.0)
        x[m < 0.1] = np.float32(-0.0)
        return x
    if kind == "far":  # quotients beyond 2^24
        return (rng.uniform(0, 1, (n, 3)) * (9e5, 500, 500)).astype(np.float32)
    return rng.uniform(-50, 80, (n, 3)).astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "edges", "tiny", "far"])
@pytest.mark.parametrize("n", [V - 1, V, V + 1, V + 2, V + 3])
def test_points_at_the_vector_threshold(ctx, oracle, n, kind):
    x = points(kind, n, np.random.default_rng(n))
    q, hil, rle = (1, n & 1, 1) if kind != "uniform" else (0, 1 - (n & 1), 0)
    for th in (0, 1024):
        want = oracle.compress(x, QN[q], 0.05, hil, rle, th, zstd=False)
        for off in (0, 1 + n % 3):
            assert container(ctx, x, off, q, 0.05, hil, rle, th) == want


@pytest.mark.parametrize("at", [0, 5, V + 1])
def test_a_point_that_is_not_finite_is_refused(ctx, xnyz, at):
    for bad in (np.nan, np.inf):
        x = points("uniform", V + 2, np.random.default_rng(3))
        x[at, at % 3] = bad
        with pytest.raises(xnyz._native.XnyzError, match="NaN or infinite"):
            container(ctx, x, 0, 1, 0.05, 1, 1, 0)
