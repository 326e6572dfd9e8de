"""The performance cases of the compress / decompress path: what a program that uses this
framework has it do, through its public entry points, from a thousand points to the 64M-point
terrain cloud of bench.py.

A case is a dict of plain values:

  op      "compress"    device points -> device container (Context.compress_device)
          "decompress"  device container -> device points (Context.decompress_device)
          "learned"     both, with the extended container whose block parameters the MLP picks
          "chunks"      host points -> zstd frames -> host points, many chunks at once
                        (Batch.roundtrip; the chunk driver's and bench.py's end-to-end path)
          "frames"      many zstd frames in device memory -> containers
                        (Context.zstd_decompress_device)
  points  points of the cloud (of each cloud for "chunks" and "frames")
  clouds  number of clouds ("chunks" and "frames": consecutive pieces of one large cloud)
  cloud   "terrain" (airborne LiDAR), "uniform" or "spheres" (clustered surfaces), the shapes of
          xnyzip_b200.synthetic_gpu; side: bounding box side
  quant   1 truncated octahedron, 0 cube;  l2: the bound;  hilbert: curve;  rle: container
"""
import math

import numpy as np
import torch

import xnyzip_b200 as X
from xnyzip_b200 import synthetic_gpu as G

DEV = "cuda:0"
LEARNED = 2  # Context.set_block_mode: block parameters by the MLP


def _case(name, op, points, cloud, side, quant, l2, hilbert, rle, clouds=1):
    return {"name": name, "op": op, "points": points, "clouds": clouds, "cloud": cloud, "side": float(side),
            "quant": quant, "l2": l2, "hilbert": hilbert, "rle": rle}


def listed():
    return [
        # the smallest clouds of the uneven batch: one call's latency, launches and waits
        _case("compress 1k", "compress", 1013, "terrain", 100, 1, 0.01, True, True),
        _case("decompress 1k", "decompress", 1013, "terrain", 100, 1, 0.01, True, True),
        # a scanned object: few cells per axis, so the container holds one curve (direct mode)
        _case("compress object 120k", "compress", 120_007, "spheres", 4, 0, 0.01, False, False),
        _case("decompress object 120k", "decompress", 120_007, "spheres", 4, 0, 0.01, False, False),
        # the reference's small plain configuration: 1M uniform points, TO 0.05, Morton, -rle
        _case("compress uniform 1M", "compress", 1_000_000, "uniform", 1000, 1, 0.05, False, True),
        _case("decompress uniform 1M", "decompress", 1_000_000, "uniform", 1000, 1, 0.05, False, True),
        # the headline: 64M terrain points at the finest bound, Hilbert, -rle
        _case("compress terrain 64M", "compress", 64_000_000, "terrain", 10000, 1, 0.001, True, True),
        _case("decompress terrain 64M", "decompress", 64_000_000, "terrain", 10000, 1, 0.001, True, True),
        # clustered surfaces as the sphere configuration has them, -normal container
        _case("compress spheres 20M", "compress", 20_000_003, "spheres", 100000, 1, 0.5, False, False),
        # extended container with learned block parameters, both directions, coarse bound
        _case("learned terrain 8M", "learned", 8_000_000, "terrain", 10000, 0, 0.1, True, True),
        # chunks of a large file end to end on host buffers, as bench.py's e2e arm cuts them
        _case("chunks 24 x 150k", "chunks", 150_000, "terrain", 480, 1, 0.01, True, True, clouds=24),
        # an archive of small clouds whose frames are already on the GPU
        _case("frames 768 x 6k", "frames", 6000, "terrain", 1000, 1, 0.01, True, True, clouds=768),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["compress", "compress", "compress", "decompress", "decompress", "decompress", "learned", "chunks",
                     "frames"])
    quant, hilbert, rle = rng.randrange(2), rng.random() < 0.5, rng.random() < 0.6
    clouds = 1
    if op == "chunks":
        points, clouds = _log_int(rng, 20_000, 200_000), rng.randint(4, 30)
    elif op == "frames":
        points, clouds = _log_int(rng, 1000, 12_000), _log_int(rng, 64, 1500)
    else:
        points = _log_int(rng, 1000, 30_000_000)
    cloud = "terrain" if op in ("chunks", "frames") else rng.choice(["terrain", "terrain", "uniform", "spheres"])
    if cloud == "terrain":
        side, l2 = math.exp(rng.uniform(math.log(10.0), math.log(1e4))), rng.choice([0.001, 0.01, 0.1])
    elif cloud == "uniform":
        side, l2 = 1000.0, rng.choice([0.01, 0.05, 0.5])
    else:
        side = math.exp(rng.uniform(math.log(4.0), math.log(1e5)))
        l2 = 0.01 if side < 100 else rng.choice([0.1, 0.5])
    return {k: v for k, v in _case("", op, points, cloud, side, quant, l2, hilbert, rle, clouds).items() if k != "name"}


def _cloud(case, seed):
    n, side = case["points"] * case["clouds"], case["side"]
    if case["cloud"] == "terrain":
        return G.gen_terrain(n, seed, DEV, extent=side, amplitude=50.0 * side / 1e4, wavelength=5000.0 * side / 1e4)
    if case["cloud"] == "uniform":
        return G.gen_uniform(n, seed, DEV).mul_(side / 1000.0)
    if side < 100:  # an object: a few large spheres
        return G.gen_spheres(n, seed, DEV, k=8, extent=side, r_median=side / 10, jitter=side / 2000)
    return G.gen_spheres(n, seed, DEV, k=max(1, n // 875), extent=side, r_median=20.0 * side / 1e5,
                         jitter=0.2 * side / 1e5)


def _seed(seed):
    return (seed * 1_000_003 + 17) & 0x7FFFFFFF


def _room(points):
    """Bytes that hold the container (or frame) of so many points in every case."""
    return 20 * points + 16384


def _context(s):
    """A context on the stream that the program's own copies go to."""
    s["stream"] = torch.cuda.Stream(DEV)
    return X.Context(0, stream=s["stream"].cuda_stream)


class _Memory:
    """Device memory that a context returned; keeps the context, whose memory it is, alive."""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3,
                                         "strides": None}


def _view(ctx, ptr, shape, typestr):
    return torch.as_tensor(_Memory(ctx, ptr, shape, typestr), device=DEV)


def prepare(case, seed):
    s = {"case": case}
    n, k = case["points"], case["clouds"]
    how = (case["quant"], case["l2"], case["hilbert"], case["rle"])
    if case["op"] in ("chunks", "frames"):
        pts = torch.split(_cloud(case, _seed(seed)).cpu(), n)
    if case["op"] == "chunks":  # a file's chunks in pinned memory, where their points go back to, and the part file
        s["batch"], s["how"] = X.Batch(0), [how] * k
        s["in"] = [p.pin_memory().numpy() for p in pts]
        s["out"] = [torch.zeros(p.shape, dtype=torch.float32).pin_memory().numpy() for p in pts]
        s["file"] = np.zeros(k * _room(n), np.uint8)
    elif case["op"] == "frames":  # the archive's frames in one device buffer, at offsets of 256 bytes
        batch, host = X.Batch(0), [p.numpy() for p in pts]
        frames = batch.compress(host, [how] * k)
        sizes = [len(f) for f in batch.compress(host, [how] * k, use_zstd=False)]
        batch.close()
        at = np.concatenate([[0], np.cumsum([-(-len(f) // 256) * 256 for f in frames])])
        packed = np.zeros(int(at[-1]), np.uint8)
        for f, a in zip(frames, at):
            packed[a:a + len(f)] = np.frombuffer(f, np.uint8)
        s["ctx"], s["frames"] = _context(s), torch.from_numpy(packed).to(DEV)
        s["out"] = torch.zeros((k, _room(n)), dtype=torch.uint8, device=DEV)
        s["args"] = ([s["frames"].data_ptr() + int(a) for a in at[:-1]], [len(f) for f in frames],
                     [s["out"].data_ptr() + i * _room(n) for i in range(k)], sizes)
    else:
        s["ctx"] = _context(s)
        if case["op"] == "learned":
            s["ctx"].set_block_mode(LEARNED)
        s["points"] = _cloud(case, _seed(seed))
        torch.cuda.synchronize()
        if case["op"] == "decompress":  # the container as a program reads it from storage: in a buffer of its own
            writer = X.Context(0)
            p, size = writer.compress_device(s["points"].data_ptr(), n, *how)
            s["container"] = _view(writer, p, (size,), "|u1").clone()
            torch.cuda.synchronize()
            writer.close()
            del s["points"]
        else:
            s["file"] = torch.zeros(_room(n), dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    q, l2, hilbert, rle = case["quant"], case["l2"], case["hilbert"], case["rle"]
    if case["op"] == "chunks":  # the frames go into the part file one after another
        frames = s["batch"].roundtrip(s["in"], s["how"], s["out"])
        at = 0
        for f in frames:
            s["file"][at:at + f.size] = f
            at += f.size
        return {"file": s["file"], "sizes": np.array([f.size for f in frames]), "points": s["out"]}
    ctx = s["ctx"]
    if case["op"] == "frames":
        return {"sizes": ctx.zstd_decompress_device(*s["args"]), "containers": s["out"]}
    if case["op"] == "decompress":
        p, n = ctx.decompress_device(s["container"].data_ptr(), s["container"].numel(), q, l2, rle)
        return {"points": _view(ctx, p, (n, 3), "<f4")}
    p, size = ctx.compress_device(s["points"].data_ptr(), case["points"], q, l2, hilbert, rle)
    with torch.cuda.stream(s["stream"]):  # the context's memory is the next call's: the program keeps a copy
        s["file"][:size].copy_(_view(ctx, p, (size,), "|u1"))
    info = ctx.last_info
    out = {"container": s["file"], "size": size, "units": info.num_units, "mse": info.mse,
           "max_l2_error": info.max_l2_error}
    if case["op"] == "learned":
        p, n = ctx.decompress_device(p, size, q, l2, rle)
        out["points"] = _view(ctx, p, (n, 3), "<f4")
    return out


def work(case):
    """12 bytes a point and the container, whose size is estimated: per point its place among the cells
    of its 128^3 block, per occupied block its id and count.  Within a third of what the coders reach."""
    n, cells = case["points"], case["side"] / case["l2"]
    dims = 3.0 if case["cloud"] == "uniform" else 2.0  # the others are surfaces
    blocks = max(1.0, (cells / 115.0) ** dims)
    occupied = blocks * -math.expm1(-n / blocks)
    bits = 5.0 + min(20.0, max(3.0, (dims + 0.2) * math.log2(max(2.0, cells)) - math.log2(n)))
    bits += occupied / n * (64.0 + math.log2(blocks))
    if case["op"] == "frames":  # zstd takes the counts' zero bytes out
        bits = min(bits, 64.0)
    points, container = 12.0 * n, n * bits / 8.0
    k = case["clouds"]
    if case["op"] == "chunks":
        return {"bytes": k * (2 * points + container), "flops": 0.0}
    if case["op"] == "frames":
        return {"bytes": k * 2 * container, "flops": 0.0}
    if case["op"] == "learned":  # points in, container out; container in, points out
        return {"bytes": 2 * (points + container), "flops": 0.0}
    return {"bytes": points + container, "flops": 0.0}


def _half_away(v):
    return np.copysign(np.floor(np.abs(v.astype(np.float64)) + 0.5), v).astype(np.float32)


def _cells(x, case):
    """Lattice cells of the points: float32 by definition (the cell is what the container codes)."""
    f = np.float32
    off = x.min(0)
    q = (x - off) / f(float(f(2.0) * f(case["l2"])) / math.sqrt(5.0 if case["quant"] else 3.0))
    if not case["quant"]:
        return np.floor(q).astype(np.int64), off
    even = _half_away(q * f(0.5)) * f(2.0)
    odd = _half_away((q - f(1.0)) * f(0.5)) * f(2.0) + f(1.0)

    def dist(c):
        d = (q - c) * (q - c)
        return d[:, 0] + (d[:, 1] + d[:, 2])

    c = np.where((dist(even) <= dist(odd))[:, None], even, odd).astype(np.int64)
    is_odd = c[:, 0] & 1
    c[:, 0] = (c[:, 0] + is_odd) >> 1
    c[:, 1] = (c[:, 1] + is_odd) >> 1
    return c, off


def _centres(c, case):
    """The cells' points in 64 bits, before the offset is added back."""
    step = 2.0 * float(np.float32(case["l2"])) / math.sqrt(5.0 if case["quant"] else 3.0)
    if not case["quant"]:
        return (c + 0.5) * step
    low = c[:, 2] & 1
    return np.stack([2 * c[:, 0] - low, 2 * c[:, 1] - low, c[:, 2]], 1) * step


def _spread(v):
    r = np.zeros_like(v)
    for b in range(21):
        r |= ((v >> b) & 1) << (3 * b)
    return r


def _morton(c):
    return _spread(c[:, 0]) | (_spread(c[:, 1]) << 1) | (_spread(c[:, 2]) << 2)


def exact(case, seed):
    """Decoded points of Morton-ordered containers and the error statistics of a compress call, in
    64 bits.  None for bytes, for the Hilbert order (its plain restatement is a search for the curve,
    not a formula), and where float32 does not resolve the bound, so that the statistics are those
    of the path's own rounding."""
    n = case["points"]
    if case["op"] in ("chunks", "frames") or n > 20_000_003:
        return None
    if case["op"] != "compress" and case["hilbert"]:
        return None
    x = _cloud(case, _seed(seed)).cpu().numpy()
    c, off = _cells(x, case)
    if c[:, 2].min() < 0:  # the reference wraps a cell below the box: no plain value
        return None
    if case["op"] == "compress":
        if case["side"] * 2.0 ** -24 * 100 > case["l2"]:
            return None
        e = (((x - off).astype(np.float64) - _centres(c, case)) ** 2).sum(1)
        return {"container": None, "size": None, "units": None, "mse": float(e.mean()),
                "max_l2_error": float(np.sqrt(e.max()))}
    if c.max() < 1024:  # direct mode: one curve over the whole cloud
        order = np.argsort(_morton(c), kind="stable")
    else:  # 128^3 super-blocks, their eight quadrants, the curve inside each
        nx, ny = c[:, 0].max() // 128 + 1, c[:, 1].max() // 128 + 1
        b = c >> 7
        quad = ((c >> 6) & 1) @ np.array([1, 2, 4])
        order = np.lexsort((_morton(c & 63), quad, b[:, 0] + nx * (b[:, 1] + ny * b[:, 2])))
    points = _centres(c[order], case) + off.astype(np.float64)
    if case["op"] == "learned":
        return {"container": None, "size": None, "units": None, "mse": None, "max_l2_error": None, "points": points}
    return {"points": points}
