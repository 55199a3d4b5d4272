"""The library's host path on a CPU: its own sources built against
fake_cudart.cc in place of the CUDA runtime (tests/_build/), for tests of
planning, workspaces, graph reuse and memory limits that need no GPU."""
import contextlib
import ctypes as C
import gc
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from morphogen_b200 import _native as N
from morphogen_b200 import build as B

HERE = Path(__file__).resolve().parent
OUT = HERE / "_build"
GIB = 1 << 30


def build() -> Path:
    """Compile what has changed; the kernels only as far as PTX, nothing runs them."""
    OUT.mkdir(exist_ok=True)
    lib, newest = OUT / "libmorphogen_fake.so", max(p.stat().st_mtime for p in B.HEADERS)
    inc = ["-I", str(B.ROOT / "include"), "-I", str(B.CSRC)]
    nv = [B.nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC"]
    cxx = ["g++", "-O1", "-std=c++17", "-fPIC", "-w", "-I", str(Path(nv[0]).resolve().parents[1] / "include")]
    jobs, objs = [], []
    for src in [*B.SOURCES, HERE / "fake_cudart.cc"]:
        obj = OUT / (src.stem + ".o")
        objs.append(obj)
        if not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, newest):
            jobs.append([*(cxx if src.suffix == ".cc" else nv), *inc, "-c", str(src), "-o", str(obj)])
    with ThreadPoolExecutor(5) as pool:
        for r in pool.map(lambda c: subprocess.run(c, capture_output=True, text=True), jobs):
            assert r.returncode == 0, r.stdout + r.stderr
    if not lib.exists() or any(o.stat().st_mtime > lib.stat().st_mtime for o in objs):
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", str(lib), *map(str, objs), "-lpthread"], check=True)
    return lib


@contextlib.contextmanager
def fake_library(path: Path):
    """`_native` bound to the fake-device library for the duration."""
    # Objects release their handles through whichever library is bound: what
    # belongs to the one goes before the other is.
    gc.collect()
    real_path, real_lib = N.LIB_PATH, N._lib
    gc.disable()
    N.LIB_PATH, N._lib = path, None
    try:
        L = N.lib()
        L.fake_reset.argtypes = [C.c_uint64, C.c_int]
        L.fake_fail.argtypes = [C.c_uint64]
        L.fake_last_delta.argtypes = [C.c_uint64 * 4]
        for f in (L.fake_used, L.fake_peak, L.fake_dead_launches, L.fake_graphs):
            f.restype = C.c_uint64
        gc.enable()
        yield L
    finally:
        gc.collect()
        gc.enable()
        N.LIB_PATH, N._lib = real_path, real_lib
