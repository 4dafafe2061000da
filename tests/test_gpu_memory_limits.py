"""Calls where device memory is short (GPU, on a build that stops at a number of
bytes): what fitted without the slots of the one-pass paths still fits, with the
same result, and a call that does not fit leaves nothing behind."""
import pytest

from memory_limit import limited_library, run_script

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def limited(built_lib, tmp_path_factory):
    return limited_library(str(tmp_path_factory.mktemp("limited")))


LIST = """
import os
import numpy as np
import irregular_gb300 as irr
from helpers import random_box
n, cut2 = 200_000, np.float32(6.25)
pos, side = random_box(n, 64 / (4.0 / 3.0 * np.pi * 2.5 ** 3), 3)
want = irr.neighbor_build(pos, float(side), float(cut2)).to_host()
nodes = n * (12 + 16 + 6 * 4 + 16)  # the raw and the converted positions, keys and places, positions in cell order
pairs, slots = 8 * len(want), 4 * n * 112
count_first = nodes + pairs + pairs // 2  # the list and its rows
lines = {  # bytes: whether the list fits
    2 * (nodes + slots + pairs): True,
    nodes + slots + pairs // 2: True,   # the slots, but not the list beside them
    count_first + (4 << 20): True,      # not the slots
    pairs + (1 << 20): False,           # the list, but not its rows
    pairs - (1 << 20): False,
    nodes // 4: False,
}
assert count_first + (4 << 20) < nodes + slots + pairs // 2 < nodes + slots + pairs
for limit, fits in list(lines.items()) * 3:
    os.environ["IRR_MEMORY_LIMIT"] = str(limit)
    try:
        got = irr.neighbor_build(pos, float(side), float(cut2))
    except irr.IrregularError as e:
        assert e.status == irr.IRR_ERR_NOMEM and not fits, (limit, e)
    else:
        assert fits, limit
        assert np.array_equal(got.to_host(), want)
        got.close()
print("done")
"""


def test_list(limited):
    assert "done" in run_script(limited, LIST)
