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


HANDLE = """
import os
import numpy as np
import irregular_gb300 as irr
from helpers import random_box
from oracle import oracle as O
n, rc = 100_000, 2.5
pos, side = random_box(n, 64 / (4.0 / 3.0 * np.pi * rc ** 3), 3)
edges = O.neighbor_half_list(pos, float(side), np.float32(rc * rc))
e = len(edges)


def handle(**cfg):
    shard = cfg.pop("shard", False)
    os.environ.pop("IRR_MEMORY_LIMIT", None)
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MOLDYN, **cfg))
    h.set_params(irr.moldyn_params(float(side), rc))
    if shard:
        h.set_shard(100, n // 2)
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    return h


def result(h):
    os.environ.pop("IRR_MEMORY_LIMIT", None)
    h.step()
    return h.get_result(elm_size=12).view(np.uint32), h.info().layout


"""

FAILED = HANDLE + """
slots = 4 * n * ((3 * e // n + 24 + 7) // 8 * 8)
for cfg, enough in ((dict(layout=irr.IRR_LAYOUT_CSR), 16 * e + 60 * n + slots + (1 << 20)),
                    (dict(exec=irr.IRR_EXEC_PLAIN), 8 * e + 50 * n), (dict(), 45 * e)):
    h = handle(**cfg)
    for limit in (8 * e + 13 * n, 8 * e + 29 * n, 8 * e + 50 * n, 15 * e) * 20:
        os.environ["IRR_MEMORY_LIMIT"] = str(limit)
        for call in (h.init, h.step):  # a step makes the set-up, or says why not
            try:
                call()
            except irr.IrregularError as err:
                assert err.status == irr.IRR_ERR_NOMEM, str(err)
            else:
                assert limit >= enough, (cfg, limit)
                h.close()
                h = handle(**cfg)
                break
        if h.info().num_edges != e:
            h.set_edges(edges)
    # nothing was lost on the way: the set-up that fits alone fits after them
    os.environ["IRR_MEMORY_LIMIT"] = str(enough)
    h.init()
    f64, sabs = O.lj_reduce_f64(pos.astype(np.float64), edges, O.lj_param(rc * rc, float(side), True))
    got = result(h)[0].view(np.float32)
    assert np.abs(got - f64).max() <= 1e-6 * np.abs(f64).max()
    h.close()
print("done")
"""


def test_failed_setup(limited):
    assert "done" in run_script(limited, FAILED)


SETUP = HANDLE + """
h = handle(layout=irr.IRR_LAYOUT_STAGED)
h.init()
st = h.staged()
h.close()
words = 4 * (len(st["words"]) + len(st["ids"]) + len(st["slice_off"])) + 32 * len(st["items"])
# without slots: the half list and the rows, records, positions, results and
# orders, a cursor per node; then the layout beside them
bare = 16 * e + (12 + 32 + 12 + 4) * n + (2 << 20)
slots = 4 * n * ((3 * e // n + 24 + 7) // 8 * 8)
sliced = 4 * 2 * e * 5 // 4
configs = {
    "auto": ({}, bare + words, bare - (2 << 20) - 4 * e),
    "staged": (dict(layout=irr.IRR_LAYOUT_STAGED), bare + words, bare - (2 << 20) - 4 * e),
    "sliced": (dict(layout=irr.IRR_LAYOUT_SLICED), bare + sliced, bare - (2 << 20) - 4 * e),
    "csr": (dict(layout=irr.IRR_LAYOUT_CSR), bare, bare - (2 << 20) - 4 * e),
    "shard": (dict(layout=irr.IRR_LAYOUT_CSR, shard=True), bare + 4 * e, bare - (2 << 20) - 4 * e),
}
for name, (cfg, least, too_little) in configs.items():
    # less than the slots take with what is made of them: the rows, or the staged layout and its scratch
    assert least < 8 * e + 44 * n + slots + (4 * e + words if name in ("auto", "staged") else 8 * e), name
    h = handle(**cfg)
    want = result(h)
    h.close()
    for limit in (4 * least, least, least, too_little, 12 * e, 8 * e + 13 * n):
        h = handle(**cfg)
        os.environ["IRR_MEMORY_LIMIT"] = str(limit)
        try:
            h.init()
        except irr.IrregularError as err:
            assert err.status == irr.IRR_ERR_NOMEM and limit < least, (name, limit, least, str(err))
            # nothing half made: no step, and the same handle once there is room
            for _ in range(3):
                try:
                    h.step()
                    raise SystemExit("a step without a set-up")
                except irr.IrregularError as again:
                    status = again.status
                    assert status in (irr.IRR_ERR_NOMEM, irr.IRR_ERR_STATE), str(again)
            os.environ.pop("IRR_MEMORY_LIMIT")
            if status == irr.IRR_ERR_STATE:  # the half list was given up
                h.set_edges(edges)
            h.init()
        else:
            assert limit >= least or name == "auto", (name, limit)
        got = result(h)
        if limit >= least:
            assert got[1] == want[1], (name, limit, got[1], want[1])
        if got[1] == want[1]:
            assert np.array_equal(got[0], want[0]), (name, limit)
        h.close()
print("done")
"""


def test_setup(limited):
    assert "done" in run_script(limited, SETUP)


RELAYOUT = HANDLE + """
star = np.stack([np.zeros(3000, np.int32), np.arange(1, 3001, dtype=np.int32)], 1)
hub = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MOLDYN))
hub.set_params(irr.moldyn_params(float(side), rc))
hub.set_edges(star)
hub.set_nodes(pos[:3001], 12)
hub.init()
assert hub.info().layout != irr.IRR_LAYOUT_STAGED
h = handle()
h.init()
assert h.info().layout == irr.IRR_LAYOUT_STAGED
want, shape = result(h)[0], (h.info().lanes_per_row, h.info().block_nodes, h.info().num_blocks)
for _ in range(5):
    b = irr.Batch(0)
    b.add(h)
    b.add(hub)
    os.environ["IRR_MEMORY_LIMIT"] = str(8 * e)  # not the rows beside the layout
    try:
        b.finalize()
        raise SystemExit("laid out without room")
    except irr.IrregularError as err:
        assert err.status == irr.IRR_ERR_NOMEM, str(err)
    got, layout = result(h)
    assert layout == irr.IRR_LAYOUT_STAGED and np.array_equal(got, want)
    assert shape == (h.info().lanes_per_row, h.info().block_nodes, h.info().num_blocks)
    b.close()
b = irr.Batch(0)
b.add(h)
b.add(hub)
b.finalize()
assert h.info().layout != irr.IRR_LAYOUT_STAGED
b.close()
print("done")
"""


def test_failed_relayout(limited):
    """The handle keeps the layout that it had."""
    assert "done" in run_script(limited, RELAYOUT)
