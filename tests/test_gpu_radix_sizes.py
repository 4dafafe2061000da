"""The radix sort at the edges of its tiles (2,048 items), groups of tiles
(65,536) and of the size up to which places are summed (8,388,608), bit for bit:
a node order against the oracle's, an entry sort against a host sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def partition(irr, pos, edges, **cfg):
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, layout=irr.IRR_LAYOUT_CSR, **cfg))
    h.set_params(irr.minimd_params(6.25))
    h.set_edges(np.ascontiguousarray(edges, np.int32))
    h.set_nodes(pos, 12)
    h.init()
    got = h.partition()
    h.close()
    return got


@pytest.mark.parametrize("n", [2, 255, 2047, 2048, 2049, 65535, 65536, 65537, 133121])
@pytest.mark.parametrize("spread", [1.0, 1e-3])
def test_node_order(built_lib, oracle_lib, n, spread):
    """spread: nodes that share keys keep their order."""
    import irregular_gb300 as irr
    O = oracle_lib
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)).astype(np.float32) * np.float32(spread)
    pos[:2] = [[0, 0, 0], [1, 1, 1]]
    edges = np.array([[0, n - 1]], np.int32)
    lo, scale = O.morton_frame(pos)
    ref_perm, _, _, _ = O.partition(pos, lo, scale, edges, curve="hilbert")
    assert np.array_equal(partition(irr, pos, edges)[0], ref_perm)


@pytest.mark.parametrize("entries", [(1 << 23) - 2, 1 << 23, (1 << 23) + 2])
def test_entry_order(built_lib, entries):
    """A hub of more than 1,024 edges: the entries are sorted by column, then row."""
    import irregular_gb300 as irr
    n = 300007
    rng = np.random.default_rng(3)
    edges = rng.integers(0, n, (entries // 2, 2)).astype(np.int32)
    edges[:2000, 0] = 5
    _, off, col = partition(irr, rng.random((n, 3)).astype(np.float32), edges, reorder=0)
    both = np.concatenate([edges, edges[:, ::-1]]).astype(np.int64)
    keys = np.sort(both[:, 0] * n + both[:, 1])
    assert np.array_equal(np.diff(off), np.bincount(both[:, 0], minlength=n))
    assert np.array_equal(col, keys % n)
