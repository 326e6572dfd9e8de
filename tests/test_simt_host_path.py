"""The host path of the library on the CPU (simt_host.py): what a failed call leaves behind, with
streams that run their work as late as they may."""
import pytest

import simt_host

PARTS = """
import struct
from oracle import Oracle
o = Oracle()

def streams(raw, rle):
    '''Container -> (head, [[meta, data], ..], tail).'''
    units, params = struct.unpack_from("<QQ", raw, 0)
    at = 16 + 4 * params + 14
    head, out = raw[:at], []
    for _ in range((2 if raw[at - 1] else 6) + rle):
        dl, ml = struct.unpack_from("<QQ", raw, at)
        out.append([raw[at + 16:at + 16 + ml], raw[at + 16 + ml:at + 16 + ml + dl]])
        at += 16 + ml + dl
    assert len(raw) == at + 12
    return head, out, raw[at:]

def joined(head, parts, tail):
    return head + b"".join(struct.pack("<QQ", len(d), len(m)) + m + d for m, d in parts) + tail
"""


@pytest.mark.parametrize("damage", ["counts too short", "quads too short", "no quad codes", "no count codes"])
def test_failed_decompress_leaves_no_work_behind(oracle, damage):
    """A stream that the host finds damaged after others have been queued: nothing may read the caller's
    container, or write the context's workspace, once the call has returned."""
    simt_host.run(PARTS + f"""
damage = {damage!r}
ctx = X.Context(0)
rng = np.random.default_rng(3)
x = rng.uniform(0, 400, (6000, 3)).astype(np.float32)
x = np.concatenate([x, x[:3000]])  # counts 1 and 2: one bit each
raw = o.compress(x, "to", 0.05, 1, 1, 0, zstd=False)
head, s, tail = streams(raw, 1)
which = 6 if "count" in damage else 5
if "short" in damage:
    if which == 5:  # eight codes of three bits
        s[5][0] = struct.pack(">I", 8) + b"".join(struct.pack(">BBI", i + 1, 3, i) for i in range(8))
    s[which][1] = s[which][1][:100]
else:
    s[which] = [struct.pack(">I", 0), b""]
bad = joined(head, s, tail)
p = device(bad)
try:
    ctx.decompress_device(p, len(bad), 1, 0.05, 1)
    raise SystemExit("accepted")
except X.XnyzError as e:
    assert e.status == 2, e
assert simt.simt_pending() == 0
simt.simt_device_free(p)
y = rng.uniform(0, 300, (5000, 3)).astype(np.float32)
for _ in range(2):
    raw = ctx.compress(y, 1, 0.05, 1, 1, use_zstd=False)
    assert raw == o.compress(y, "to", 0.05, 1, 1, zstd=False)
    assert ctx.decompress(raw, 1, 0.05, 1, is_zstd=False).tobytes() == o.decompress(raw, "to", 0.05, 1, zstd=False).tobytes()
    no_fault()
""")


def test_sort_after_a_failed_allocation(oracle):
    """The sort's status words cannot grow for a large cloud: that call fails, and the next smaller one,
    for which the old words sufficed, allocates its own."""
    simt_host.run(PARTS + """
ctx = X.Context(0)
rng = np.random.default_rng(3)
x = rng.uniform(0, 300, (60_000, 3)).astype(np.float32)

def same(n):
    raw = ctx.compress(x[:n], 1, 0.05, 1, 1, use_zstd=False)
    no_fault()
    assert raw == o.compress(x[:n], "to", 0.05, 1, 1, zstd=False)

same(9000)
try:  # grows the workspace: 128 KB a frame
    ctx.zstd_decompress_device([device(b"no frame")] * 100, [8] * 100, [device(bytes(8))] * 100, [8] * 100)
except X.XnyzError:
    pass
simt.simt_malloc_limit(100_000)
try:
    ctx.compress(x, 1, 0.05, 1, 1, use_zstd=False)
    raise SystemExit("allocated")
except X.XnyzError as e:
    assert e.status == 4, e
simt.simt_malloc_limit(1 << 40)
same(9000)
same(60_000)
""")


@pytest.mark.parametrize("rle,threshold", [(1, 0), (0, 0), (0, 1024)])
def test_streams_whose_waits_run_out(oracle, rle, threshold):
    """The stream decoders' status words get lost, so that every block but the first waits in vain
    (64 times instead of seconds): the streams are decoded by one thread, and the result is right."""
    simt_host.run(PARTS + f"""
ctx = X.Context(0)
x = np.random.default_rng(9).uniform(0, 40, (30_000, 3)).astype(np.float32)
raw = o.compress(x, "to", 0.05, 1, {rle}, {threshold}, zstd=False)
want = o.decompress(raw, "to", 0.05, {rle}, zstd=False).tobytes()
simt.simt_drop_status(b"decode_sync_kernel")
assert ctx.decompress(raw, 1, 0.05, {rle}, is_zstd=False).tobytes() == want
kernels = simt.simt_kernels().decode()
assert "decode_sequential_kernel" in kernels, kernels
simt.simt_drop_status(b"")
simt.simt_clear()
assert ctx.decompress(raw, 1, 0.05, {rle}, is_zstd=False).tobytes() == want
assert "decode_sequential_kernel" not in simt.simt_kernels().decode()
no_fault()
""")


@pytest.mark.parametrize("where", ["device", "pinned", "peer"])
@pytest.mark.parametrize("n", [200, 6000])
def test_containers_that_only_a_copy_can_reach(oracle, where, n):
    """decompress_device takes containers in any memory that a copy can read: another device's without
    peer access (whose addresses hold other bytes for a kernel here), pinned host memory."""
    simt_host.run(PARTS + f"""
ctx = X.Context(0)
x = np.random.default_rng({n}).uniform(0, 60, ({n}, 3)).astype(np.float32)
raw = o.compress(x, "to", 0.05, 1, 1, 0, zstd=False)
p = dict(device=lambda: device(raw), pinned=lambda: device(raw, pinned=True), peer=lambda: peer(raw))[{where!r}]()
q, k = ctx.decompress_device(p, len(raw), 1, 0.05, 1)
no_fault()
assert ctypes.string_at(q, 12 * k) == o.decompress(raw, "to", 0.05, 1, zstd=False).tobytes()
""")
