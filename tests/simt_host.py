"""The library's sources, kernels included, compiled for the CPU against tests/simt (fibers for the
threads of a block, streams that run as late as they may), so that faults that must not be shown on a
GPU are shown here: missing barriers, work left queued by a failed call, failed allocations.

    lib = simt_host.library()          # path of the shared library
    simt_host.run(script)              # runs `script` in a process where xnyzip_b200 is that library
"""
import concurrent.futures as cf
import functools
import glob
import hashlib
import os
import re
import shutil
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "xnyzip_b200", "csrc")
SIMT = os.path.join(HERE, "simt")
CXX = "/usr/bin/g++"

# inline assembly, and the text in whose place it stands
ASM = [
    (r'asm\("mov\.u32 %0, %%lanemask_lt;" : "=r"\(m\)\);', "m = (1u << simt::lane()) - 1u;"),
    (r'asm volatile\("st\.relaxed\.gpu\.global\.b128 [^;]*;" ::"l"\(p\), "q"\(x\) : "memory"\);',
     "if (!simt::dropped()) *p = x;"),
    (r'asm volatile\("ld\.relaxed\.gpu\.global\.b128 [^;]*;" : "=q"\(x\) : "l"\(p\) : "memory"\);', "x = *p;"),
    (r'asm volatile\("cp\.async\.cg\.shared\.global [^;]*;" ::[^;]*\);', "std::memcpy(smem, g, 16);"),
    (r'asm volatile\("cp\.async\.wait_all;" ::: "memory"\);', ""),
    (r'asm volatile\("\{ \.reg \.pred q; setp[^}]*\}"\s*:[^;]*\);', "v = ok ? *p : 0ull;"),
    (r'asm volatile\("prmt\.b32 [^;]*;" :[^;]*\);', "d = __byte_perm((u32)key, (u32)(key >> 32), sel);"),
    (r'asm\("\{ \.reg \.pred p; and\.b32.*?: "r"\(d\), "r"\(1u << b\)\);',
     "{ const bool x = (d >> b) & 1u; m = __ballot_sync(kFullMask, x); if (!x) m = ~m; }"),
    (r'asm volatile\("bar\.sync 1, 96;" ::: "memory"\);', "simt::named_barrier(1, 96);"),
    (r'if \(near\) asm volatile\("prefetch[^;]*;" ::[^;]*;\s*else asm volatile\("prefetch[^;]*;" ::[^;]*;', ";"),
]
LAUNCH = re.compile(r"([A-Za-z_]\w*(?:<[^<>;()]*>)?)\s*<<<(.+?)>>>\((.*?)\);", re.S)


def translate(text, spin_limit):
    for pattern, to in ASM:
        text = re.sub(pattern, lambda m: to, text, flags=re.S)
    text = re.sub(r"extern __shared__ __align__\(16\) unsigned char (\w+)\[\];",
                  r"unsigned char* \1 = static_cast<unsigned char*>(simt::dynamic_shared());", text)
    text = text.replace("kSpinLimit = 1u << 23", f"kSpinLimit = {spin_limit}u").replace(")clock()", ")simt::ticks()")
    return LAUNCH.sub(lambda m: f'simt::launch("{m.group(1)}", simt::config({m.group(2)}), {m.group(1)}, {m.group(3)});', text)


@functools.lru_cache(maxsize=None)
def library(spin_limit=64, flags=("-O1",)):
    """Builds the library (once per state of the sources) and returns its path."""
    sources = sorted(glob.glob(os.path.join(CSRC, "**", "*"), recursive=True) + glob.glob(os.path.join(SIMT, "*")) +
                     [os.path.join(ROOT, "include", "xnyz.h"), __file__])
    h = hashlib.sha256(repr((spin_limit, flags)).encode())
    for s in sources:
        if os.path.isfile(s):
            with open(s, "rb") as f:
                h.update(f.read())
    base = os.path.join(tempfile.gettempdir(), f"xnyz_simt_{os.getuid()}")
    out = os.path.join(base, h.hexdigest()[:16])
    so = os.path.join(out, "libxnyz.so")
    if os.path.exists(so):
        return so
    os.makedirs(base, exist_ok=True)
    work = tempfile.mkdtemp(dir=base)
    os.makedirs(os.path.join(work, "xnyzip_b200", "csrc", "host"))
    os.makedirs(os.path.join(work, "include"))
    shutil.copy(os.path.join(ROOT, "include", "xnyz.h"), os.path.join(work, "include"))
    units = [os.path.join(SIMT, "simt.cpp")]
    for s in sources:
        name = os.path.relpath(s, CSRC)
        if name.startswith("..") or not os.path.isfile(s) or name == "k_mlp.cu":
            continue
        with open(s) as f:
            text = f.read()
        to = os.path.join(work, "xnyzip_b200", "csrc", name)
        if name.endswith((".cu", ".cuh")):
            text = translate(text, spin_limit)
        if name.endswith(".cu"):
            to += ".cpp"
        with open(to, "w") as f:
            f.write(text)
        if to.endswith(".cpp"):
            units.append(to)
    stub = os.path.join(work, "mlp.cpp")
    with open(stub, "w") as f:  # the network's kernels (tensor cores) have no host form
        f.write('#include "kernels.h"\nnamespace xnyz { namespace dev {\n'
                "void launch_mlp_forward(const float*, const float*, uint64_t, uint8_t*, uint8_t*, float*, float*, cudaStream_t) {}\n"
                "size_t mlp_gather_floats(uint64_t) { return 0; }\n"
                "void launch_mlp_train(const float*, const float*, const uint8_t*, const uint8_t*, const uint32_t*, uint64_t, uint64_t,"
                " float, float*, float*, float*, cudaStream_t) {}\n"
                "void launch_mlp_adam(float*, float*, float*, float*, float, int, cudaStream_t) {}\n}}\n")
    units.append(stub)

    def compile_one(u):
        o = os.path.join(work, os.path.basename(u) + ".o")
        r = subprocess.run([CXX, "-std=c++20", *flags, "-ffp-contract=off", "-fPIC", "-w", "-include", "cuda_runtime.h", "-I", SIMT,
                            "-I", os.path.join(work, "xnyzip_b200", "csrc"), "-c", u, "-o", o], capture_output=True, text=True)
        if r.returncode:
            raise RuntimeError(f"{u}:\n{r.stderr[:4000]}")
        return o
    with cf.ThreadPoolExecutor(os.cpu_count()) as ex:
        objects = list(ex.map(compile_one, units))
    subprocess.run([CXX, "-shared", *flags, "-Wl,-Bsymbolic", "-o", os.path.join(work, "libxnyz.so"), *objects, "-ldl"],
                   check=True)
    for o in objects:
        os.remove(o)
    try:
        os.rename(work, out)
    except OSError:  # another process was first
        shutil.rmtree(work)
    return so


PRELUDE = """
import ctypes, sys
sys.path[:0] = [{root!r}, {root!r} + "/oracle", {root!r} + "/tests"]
_real = ctypes.CDLL
simt = _real({so!r})
ctypes.CDLL = lambda p, *a, **k: simt if str(p).endswith("libxnyz.so") else _real(p, *a, **k)
import numpy as np
import xnyzip_b200 as X
ctypes.CDLL = _real
simt.simt_fault.restype = simt.simt_kernels.restype = ctypes.c_char_p
simt.simt_pending.restype = simt.simt_barriers.restype = ctypes.c_uint64
simt.simt_peer_alloc.restype = ctypes.c_void_p
simt.simt_peer_alloc.argtypes = [ctypes.c_uint64, ctypes.c_void_p]
simt.simt_device_alloc.restype = simt.simt_pinned_alloc.restype = ctypes.c_void_p
simt.simt_device_alloc.argtypes = simt.simt_pinned_alloc.argtypes = simt.simt_malloc_limit.argtypes = [ctypes.c_uint64]
simt.simt_device_free.argtypes = [ctypes.c_void_p]

def device(data, pinned=False):
    data = bytes(data) if not hasattr(data, "tobytes") else data.tobytes()
    p = (simt.simt_pinned_alloc if pinned else simt.simt_device_alloc)(len(data))
    ctypes.memmove(p, data, len(data))
    return p

def peer(data):
    at = ctypes.c_void_p()
    p = simt.simt_peer_alloc(len(data), ctypes.byref(at))
    ctypes.memmove(at, data, len(data))
    return p

def no_fault():
    assert not simt.simt_fault(), simt.simt_fault().decode()
"""


def run(script, so=None, env=None):
    """Runs the script in a new interpreter; returns its output, or raises with it."""
    code = PRELUDE.format(root=ROOT, so=so or library()) + script
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env={**os.environ, **(env or {})})
    if r.returncode:
        raise AssertionError(f"exit {r.returncode}\n{r.stdout[-2000:]}\n{r.stderr[-4000:]}")
    return r.stdout
