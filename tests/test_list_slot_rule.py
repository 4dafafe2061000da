"""The slots per node of the one-pass neighbour search (csrc/irr_list_rule.h):
none where their number, or the number of all of them, is beyond the path, so
that no search is made in vain."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG


def want(sphere, n, most):
    if not sphere < most:
        return 0
    cap = (int(1.35 * sphere) + 31) // 8 * 8
    return cap if cap <= most and cap * n < 2 ** 32 else 0


def test_rule(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    cases = [(s, n) for s in (0.0, 0.5, 7.9, 64.0, 79.3, 250.0, 735.0, 736.0, 740.0, 1023.9, 1024.0, 5e9, float("nan"))
             for n in (2, 1000, 38_347_922, 38_347_923, 100_000_000, 2 ** 31 - 1)]
    assert want(64.0, 38_347_922, 1024) == 112 and want(64.0, 38_347_923, 1024) == 0
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cmath>\n#include <cstdio>\n#include "irr_list_rule.h"\nint main()\n{\n' + "".join(
        f"    std::printf(\"%u\\n\", irr::list_slots({'NAN' if s != s else repr(s)}, {n}, 1024));\n" for s, n in cases) + "}\n")
    exe = str(tmp_path / "rule")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-I", os.path.join(PKG, "csrc"), str(src), "-o", exe], check=True)
    got = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert [int(x) for x in got] == [want(s, n, 1024) for s, n in cases]
