"""Which node records a kernel reads where they lie (csrc/irr_records.h) and
which go through the staging copy: another GPU's memory, host memory, another
address on the device, a misaligned address, a range that ends too soon."""
import shutil
import subprocess

import os
import pytest

from conftest import PKG

OWN = dict(device=1, managed=0, ordinal=0, address=4096, start=4096, size=24000)
# name: (address, record bytes, bytes in all, handle's device, what the driver says, in place)
CASES = {
    "own": (4096, 12, 24000, 0, {}, True),
    "own_24": (4096, 24, 24000, 0, {}, True),
    "inside": (4096 + 48, 12, 12000, 0, dict(address=4096 + 48), True),
    "to_the_end": (4096 + 12000, 12, 12000, 0, dict(address=4096 + 12000), True),
    "one_past_the_end": (4096 + 12000, 12, 12001, 0, dict(address=4096 + 12000), False),
    "too_long": (4096, 12, 24012, 0, {}, False),
    "longer_than_any": (4096, 12, 2 ** 64 - 1, 0, {}, False),
    "other_gpu": (4096, 12, 24000, 0, dict(ordinal=1), False),
    "other_handle": (4096, 12, 24000, 1, {}, False),
    "managed": (4096, 12, 24000, 0, dict(managed=1, ordinal=1), True),
    "managed_too_long": (4096, 12, 24012, 0, dict(managed=1), False),
    "host": (4096, 12, 24000, 0, dict(device=0), False),
    "other_address": (4096, 12, 24000, 0, dict(address=8192), False),
    "unknown_range": (4096, 12, 24000, 0, dict(start=0, size=0), False),
    "before_the_range": (4096, 12, 24000, 0, dict(start=5000), False),
    "byte_2": (4098, 12, 1200, 0, dict(address=4098), False),
    "byte_4_of_12": (4100, 12, 1200, 0, dict(address=4100), True),
    "byte_4_of_24": (4100, 24, 1200, 0, dict(address=4100), False),
    "byte_8_of_24": (4104, 24, 1200, 0, dict(address=4104), True),
    "byte_8_of_16": (4104, 16, 1600, 0, dict(address=4104), False),
    "byte_16_of_16": (4112, 16, 1600, 0, dict(address=4112), True),
}


def test_rule(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    lines = []
    for name, (p, elm, size, device, facts, want) in CASES.items():
        f = {**OWN, **facts}
        lines.append(f'    check("{name}", {p}ull, {elm}, {size}ull, {device}, {{{"true" if f["device"] else "false"}, '
                     f'{"true" if f["managed"] else "false"}, {f["ordinal"]}, {f["address"]}ull, {f["start"]}ull, '
                     f'{f["size"]}ull}}, {"true" if want else "false"});')
    src = tmp_path / "rule.cpp"
    src.write_text('''#include <cstdio>
#include "irr_records.h"
int bad = 0;
void check(const char* name, uint64_t p, int elm, uint64_t bytes, int device, irr::PointerFacts f, bool want)
{
    if (irr::records_in_place(p, elm, bytes, device, f) != want) {
        bad++;
        std::puts(name);
    }
}
int main()
{
''' + "\n".join(lines) + "\n    return bad;\n}\n")
    exe = str(tmp_path / "rule")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(PKG, "csrc"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
