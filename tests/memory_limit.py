"""A build of the library that takes at most $IRR_MEMORY_LIMIT bytes of device
memory (csrc/irr_partition.cu, IRR_MEMORY_LIMIT), and scripts run on it in a
process of their own."""
from __future__ import annotations

import os
import subprocess
import sys

from conftest import PKG, ROOT


def limited_library(tmp_dir) -> str:
    """The one translation unit compiled again, linked with the library's other objects."""
    import build as pkg_build
    pkg_build.build()
    src = os.path.join(pkg_build.CSRC, "irr_partition.cu")
    obj, lib = os.path.join(tmp_dir, "irr_partition.cu.o"), os.path.join(tmp_dir, "libirregular_limited.so")
    others = [os.path.join(pkg_build.BUILD, os.path.basename(s) + ".o") for s in pkg_build.sources() if s != src]
    for cmd in ([pkg_build.nvcc()] + pkg_build.NVCC_FLAGS + ["-DIRR_MEMORY_LIMIT", "-c", src, "-o", obj],
                [pkg_build.nvcc()] + pkg_build.ARCH + ["-shared", "-o", lib, obj] + others + ["-lcudart"]):
        out = subprocess.run(cmd, capture_output=True, text=True)
        assert out.returncode == 0, out.stdout + out.stderr
    return lib


def run_script(lib: str, script: str, timeout: int = 300) -> str:
    """The script's output; it fails with the script."""
    env = dict(os.environ, IRR_LIBRARY=lib,
               PYTHONPATH=os.pathsep.join([ROOT, PKG, os.path.join(ROOT, "tests")]))
    out = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=timeout)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout
