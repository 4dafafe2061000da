"""The edge list's check (GPU) around its tiles of 64 edges: an id out of range
at either end of a tile and of the list, and the order of idx0 across them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 63, 64, 65, 127, 128, 129, 1000]


def handle(irr, n, edges):
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, layout=irr.IRR_LAYOUT_CSR))
    h.set_params(irr.minimd_params(6.25))
    h.set_edges(np.ascontiguousarray(edges, np.int32))
    h.set_nodes(np.random.default_rng(1).random((n, 3)).astype(np.float32), 12)
    return h


def sorted_edges(n, e):
    edges = np.random.default_rng(e).integers(0, n, (e, 2))
    return edges[np.argsort(edges[:, 0], kind="stable")]


@pytest.mark.parametrize("e", SIZES)
def test_out_of_range(built_lib, e):
    import irregular_gb300 as irr
    n = 50
    for at in sorted({k for k in (0, 1, 62, 63, 64, 65, e - 2, e - 1) if 0 <= k < e}):
        for side in (0, 1):
            for bad in (-1, n, 2 ** 31 - 1):
                edges = sorted_edges(n, e)
                edges[at, side] = bad
                h = handle(irr, n, edges)
                with pytest.raises(irr.IrregularError):
                    h.init()
                h.close()


@pytest.mark.parametrize("e", SIZES)
def test_rows(built_lib, e):
    """Sorted, and with one pair of neighbours in the list exchanged."""
    import irregular_gb300 as irr
    n = 50
    for at in [None] + sorted({k for k in (0, 62, 63, 64, e - 2) if 0 <= k < e - 1}):
        edges = sorted_edges(n, e)
        if at is not None:
            edges[[at, at + 1]] = edges[[at + 1, at]]
        h = handle(irr, n, edges)
        h.init()
        _, off, col = h.partition()
        both = np.concatenate([edges, edges[:, ::-1]])
        both = both[np.lexsort((both[:, 1], both[:, 0]))]
        assert np.array_equal(np.diff(off), np.bincount(both[:, 0], minlength=n))
        assert np.array_equal(col, both[:, 1])
        h.close()
