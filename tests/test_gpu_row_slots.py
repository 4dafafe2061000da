"""Rows filled into slots (lists sorted by idx0) against the counting fill and
the oracle's partition, bit for bit: runs that end where nodes have no edges,
rows longer than the slots from either side, repeated pairs and self edges."""
import numpy as np
import pytest

from helpers import random_box

pytestmark = pytest.mark.gpu


def lists(O):
    rng = np.random.default_rng(3)
    pos, side = random_box(3000, 64.0 / (4.0 / 3.0 * np.pi * 2.5 ** 3), 21)
    box = O.neighbor_half_list(pos, float(side), np.float32(6.25))
    n = len(pos)
    hub = np.arange(n - 1, dtype=np.int32)
    some = box[(box[:, 0] % 5 != 0) & (box[:, 1] % 5 != 0)]
    twice = np.concatenate([box, box[::3], np.stack([hub[::7], hub[::7]], 1)])
    by0 = lambda e: e[np.argsort(e[:, 0], kind="stable")]
    return pos, {
        "sorted": box,
        "one_edge": box[:1],
        "last_node": np.array([[n - 1, 0]], np.int32),
        "gaps": some,
        "repeats": by0(twice),
        "unsorted": box[rng.permutation(len(box))],
        "nearly_sorted": np.concatenate([box[1:], box[:1]]),
        "hub_forward": by0(np.concatenate([box, np.stack([np.full(500, 7), hub[:500]], 1)])),
        "hub_backward": by0(np.concatenate([box, np.stack([hub[:500], np.full(500, n - 1)], 1)])),
        "long_hub": by0(np.concatenate([box, np.stack([hub, np.full(n - 1, n - 1)], 1)])),
    }


NAMES = ["sorted", "one_edge", "last_node", "gaps", "repeats", "unsorted", "nearly_sorted", "hub_forward",
         "hub_backward", "long_hub"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("reorder", [1, 0])
def test_rows_bit_exact(built_lib, oracle_lib, name, reorder):
    import irregular_gb300 as irr
    O = oracle_lib
    pos, all_lists = lists(O)
    assert sorted(all_lists) == sorted(NAMES)
    edges = np.ascontiguousarray(all_lists[name], np.int32)
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=reorder))
    h.set_params(irr.minimd_params(6.25))
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    h.init()
    perm, row_off, col = h.partition()
    if reorder:
        lo, scale = O.morton_frame(pos)
        ref_perm, _, ref_off, ref_col = O.partition(pos, lo, scale, edges, curve="hilbert")
        assert np.array_equal(perm, ref_perm)
    else:
        both = np.concatenate([edges, edges[:, ::-1]])
        both = both[np.lexsort((both[:, 1], both[:, 0]))]
        ref_col = both[:, 1]
        ref_off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=len(pos)))])
        assert np.array_equal(perm, np.arange(len(pos)))
    assert np.array_equal(row_off, ref_off)
    assert np.array_equal(col, ref_col)
    h.close()
