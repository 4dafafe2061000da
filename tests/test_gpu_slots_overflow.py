"""A list sorted by idx0 with a few rows longer than the partitioner's slots,
found in the midst of the fill while most warps are still to start (GPU): the
rows, filled again the other way, are those of the list, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hubs", [(300_000, 1), (300_005, 30), (40_009, 5)])
def test_overflow_while_warps_start(built_lib, n, hubs):
    import irregular_gb300 as irr
    rng = np.random.default_rng(n + hubs)
    i = np.repeat(np.arange(n), 6)
    edges = np.stack([i, rng.integers(0, n, i.size)], 1)
    hub = np.repeat(rng.choice(n, hubs, replace=False), 200)
    other = rng.integers(0, n, hub.size)
    ends = np.where(rng.random(hub.size) < 0.5, 1, -1)[:, None]  # long from either side
    more = np.where(ends > 0, np.stack([hub, other], 1), np.stack([other, hub], 1))
    edges = np.concatenate([edges, more])
    edges = np.ascontiguousarray(edges[np.argsort(edges[:, 0], kind="stable")], np.int32)
    both = np.concatenate([edges, edges[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    pos = rng.random((n, 3)).astype(np.float32)
    for layout in (irr.IRR_LAYOUT_CSR, irr.IRR_LAYOUT_SLICED, irr.IRR_LAYOUT_CSR):
        h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, layout=layout))
        h.set_params(irr.minimd_params(6.25))
        h.set_edges(edges)
        h.set_nodes(pos, 12)
        h.init()
        _, row_off, col = h.partition()
        assert np.array_equal(row_off, off)
        assert np.array_equal(col, both[:, 1])
        h.close()
