"""A build and what follows it in the same process, in a copy of the tree that has the compiled kernels and no more."""
import shutil
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from mlx_flashattention_steel_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent
PKG = "mlx_flashattention_steel_b200"

# the extension is what every front-end module calls, and takes or gives back calls
BOUND = f"""
import {PKG} as fa
from {PKG} import _lib, attention, kv_cache, rope
assert attention._H is kv_cache._H is rope._H is _lib.host_calls
for name in ("fwd", "bwd", "decode", "rope", "append"):
    assert getattr(_lib.host_calls, name) is getattr(sys.modules["{PKG}._host_calls"], name), name
assert _lib.host_calls.fwd() is None
"""


@pytest.fixture
def tree(tmp_path):
    """The sources, libb200fa.so and the objects, as a copy keeps them; no host extension."""
    for d in (f"{PKG}/csrc", f"{PKG}/build", f"{PKG}/integrations", "include", "oracle"):
        shutil.copytree(ROOT / d, tmp_path / d, ignore=shutil.ignore_patterns("__pycache__"))
    for f in [*(ROOT / PKG).glob("*.py"), ROOT / PKG / "libb200fa.so", ROOT / "__graft_entry__.py"]:
        shutil.copy2(f, tmp_path / f.relative_to(ROOT))
    return tmp_path


def _python(tree, code):
    r = subprocess.run([sys.executable, "-c", "import sys\n" + code], cwd=tree, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return r


def test_first_build_and_use_in_one_process(tree):
    _python(tree, f"""
import {PKG} as fa, torch
q = torch.zeros(1, 2, 64, 64, dtype=torch.float16)
try:
    fa.flash_attention(q, q, q)             # before the build: the Python code has the call
except RuntimeError as e:
    assert "no CPU path" in str(e)
import __graft_entry__
__graft_entry__.build()
""" + BOUND)


BUILD = f"from {PKG} import build\nbuild.build()\n"


@pytest.mark.parametrize("what", ["does not load", "built for another torch"])
def test_a_build_replaces_an_extension_that_is_not_for_this_torch(tree, what):
    """Newer than its sources in both cases, so that its age does not show it; the compiler has arguments of its own."""
    so, abi = tree / PKG / "_host_calls.so", tree / PKG / "build" / "_host_calls.abi"
    if what == "does not load":
        so.write_bytes(b"\x7fELF of another machine")
        abi.write_text(_lib.host_abi())
    else:
        ours, other = torch.__version__, "9" * len(torch.__version__)
        so.write_bytes((ROOT / PKG / "_host_calls.so").read_bytes().replace(b"torch " + ours.encode(), b"torch " + other.encode()))
        abi.write_text(_lib.host_abi().replace(ours, other))
    # the Python code has the calls until then, and says what is wrong
    r = _python(tree, f"from {PKG} import _lib\nlib = _lib.load()\nassert lib.b200fa_version() and _lib.host_calls.fwd() is None")
    assert "does not load" in r.stderr and f"python -m {PKG}.build" in r.stderr
    assert what == "does not load" or "built for torch 9" in r.stderr
    build = f"import os\nos.environ['CXX'] = 'env LANG=C g++'\nfrom {PKG} import build\nbuild.build()\n"
    _python(tree, build + BOUND)
    before = so.stat().st_mtime_ns
    _python(tree, build + BOUND)            # and once is enough
    assert so.stat().st_mtime_ns == before
