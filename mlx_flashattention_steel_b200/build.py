"""Builds libb200fa.so in-tree with nvcc for sm_100a, and _host_calls.so, the native half of the Python front end.

Run as ``python -m mlx_flashattention_steel_b200.build``.  Each ``csrc/*.cu`` is
compiled to an object (in parallel, skipped when newer than its sources) and
linked into ``mlx_flashattention_steel_b200/libb200fa.so`` beside this file, so
the library ships with the source tree rather than through a JIT cache.
"""
from __future__ import annotations

import concurrent.futures
import os
import shlex
import shutil
import subprocess
import sys
from pathlib import Path

from . import _lib

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libb200fa.so"
HOST = PKG / "_host_calls.so"
HOST_ABI = OBJ / "_host_calls.abi"      # what the extension beside the library was built for

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libb200fa.so cannot be built")
    return exe


def _newest_header() -> float:
    hdrs = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list((PKG.parent / "include").glob("*.h"))
    return max(h.stat().st_mtime for h in hdrs)


def _compile(src: Path, verbose: bool) -> Path:
    obj = OBJ / (src.stem + ".o")
    newest = max(src.stat().st_mtime, _newest_header())
    if obj.exists() and obj.stat().st_mtime > newest:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        sys.stderr.write(res.stderr)
    return obj


def _build_host_calls(force: bool) -> None:
    """The native half of the Python front end: an extension module against the installed torch, beside the library.  Built again
    when its sources, that torch or that Python are others than it was built with, or when it does not load."""
    import sysconfig

    import torch

    src = CSRC / "host_calls.cpp"
    newest = max(src.stat().st_mtime, (PKG.parent / "include" / "b200fa.h").stat().st_mtime)
    built_for = _lib.host_abi()
    if (HOST.exists() and not force and HOST.stat().st_mtime > newest and HOST_ABI.exists() and HOST_ABI.read_text() == built_for
            and _lib.host_calls.bind()):
        return
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    new = HOST.with_suffix(f".{os.getpid()}.tmp")
    cmd = [*shlex.split(os.environ.get("CXX", "g++")), "-O2", "-std=c++17", "-shared", "-fPIC",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DB200FA_HOST_ABI="{built_for}"',
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}",
           f"-I{cuda}/include", str(src), "-o", str(new), f"-L{PKG}", "-lb200fa", f"-L{root}/lib", "-ltorch_python",
           "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    try:
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"building {HOST.name} failed:\n{res.stdout}\n{res.stderr}")
        os.replace(new, HOST)
    finally:
        new.unlink(missing_ok=True)
    HOST_ABI.write_text(built_for)
    _lib.host_calls.error = None        # if importing it failed in this process: try again


def build(verbose: bool = False, force: bool = False) -> Path:
    OBJ.mkdir(exist_ok=True)
    srcs = sorted(CSRC.glob("*.cu"))
    if force:
        for o in OBJ.glob("*.o"):
            o.unlink()
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    if (not LIB.exists()) or force or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        cmd = [_nvcc(), "-shared", "-o", str(LIB), *map(str, objs)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _build_host_calls(force)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
