"""In-tree build of the native library: plain ``nvcc`` for sm_100a, no torch headers.

Every ``.cu`` under ``csrc/`` is compiled to an object (in parallel, cached by
source hash) and linked into ``zen_repro_b200/_lib/libzen_b200.so``, which the
Python side opens through ``csrc/fastcall.c``.  The kernels take raw device pointers and a
stream, so the library has no dependency on libtorch and builds in seconds.

    python -m zen_repro_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIBDIR = PKG / "_lib"
LIBNAME = "libzen_b200.so"
CALLNAME = "zen_fastcall.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found")
    return exe


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _digest(src: Path) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    h.update(src.read_bytes())
    for hdr in sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")):
        h.update(hdr.read_bytes())
    return h.hexdigest()[:16]


def _compile_one(src: Path, verbose: bool) -> tuple[Path, str]:
    obj = LIBDIR / f"{src.stem}.{_digest(src)}.o"
    log = ""
    if not obj.exists():
        for old in LIBDIR.glob(f"{src.stem}.*.o"):
            old.unlink()
        cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        log = r.stdout + r.stderr
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{log}")
        (LIBDIR / f"{src.stem}.ptxas.log").write_text(log)
    return obj, log


def _fastcall_want() -> str:
    """What ``fastcall.stamp`` says beside an extension that belongs to this source and this interpreter."""
    return hashlib.sha256((CSRC / "fastcall.c").read_bytes()).hexdigest() + sys.version


def fastcall_current() -> bool:
    """Whether the CPython extension is there and was built from this source for this interpreter: one that another Python
    built can be opened all the same, and then runs with the wrong object layouts."""
    stamp = LIBDIR / "fastcall.stamp"
    return (LIBDIR / CALLNAME).exists() and stamp.exists() and stamp.read_text() == _fastcall_want()


def build_fastcall() -> Path:
    """The small CPython extension through which Python calls the library's functions."""
    src, out, stamp = CSRC / "fastcall.c", LIBDIR / CALLNAME, LIBDIR / "fastcall.stamp"
    if not fastcall_current():
        LIBDIR.mkdir(exist_ok=True)
        cc = shutil.which("gcc") or shutil.which("cc")
        if cc is None:
            raise RuntimeError("no C compiler found")
        tmp = out.with_suffix(f".{os.getpid()}.tmp")          # ranks that start together each replace the file as a whole
        cmd = [cc, "-O2", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], str(src), "-o", str(tmp)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("fastcall build failed:\n" + r.stdout + r.stderr)
        os.replace(tmp, out)
        stamp.write_text(_fastcall_want())
    return out


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile and link the native library; returns the path of the ``.so``."""
    LIBDIR.mkdir(exist_ok=True)
    if force:
        for f in LIBDIR.glob("*.o"):
            f.unlink()
    build_fastcall()
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs) or 1)) as ex:
        results = list(ex.map(lambda s: _compile_one(s, verbose), srcs))
    objs = [o for o, _ in results]
    out = LIBDIR / LIBNAME
    stamp = LIBDIR / "link.stamp"
    want = " ".join(o.name for o in objs)
    if force or not out.exists() or not stamp.exists() or stamp.read_text() != want:
        cmd = [_nvcc(), "-shared", "-o", str(out), *map(str, objs), "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
        stamp.write_text(want)
    if verbose:
        for _, log in results:
            if log:
                print(log)
    return out


def lib_path() -> Path:
    return LIBDIR / LIBNAME


def fastcall_path() -> Path:
    return LIBDIR / CALLNAME


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(p)
