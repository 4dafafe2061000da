"""The staged layout's cut refused in the midst of its launch (GPU): a graph of
many runs, a few of whose blocks touch more nodes than a narrow table holds, so
that the refusal is raised while most CTAs are still to start.  AUTO then takes
the wide limits, whose layout equals the oracle's bit for bit, and an explicit
IRR_LAYOUT_STAGED refuses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDE = dict(slices_per_item=8, tab_max=1008, stream_max=6400)


def pocketed(n, pockets, seed):
    """Pairs (i, i + 1 .. i + 4), and per pocket a block of 8 rows with 100
    partners of their own each (808 ids: above 640, below 1008)."""
    i = np.repeat(np.arange(n), 4)
    chain = np.stack([i, i + np.tile(np.arange(1, 5), n)], 1)
    first = 8 * np.sort(np.random.default_rng(seed).choice(n // 8 - 200, pockets, replace=False))
    k = np.arange(8)
    a = (first[:, None, None] + k[None, :, None] + np.zeros((1, 1, 100), np.int64)).ravel()
    b = (first[:, None, None] + 16 + 100 * k[None, :, None] + np.arange(100)[None, None, :]).ravel()
    e = np.concatenate([chain[chain[:, 1] < n], np.stack([a, b], 1)])
    return np.unique(e, axis=0).astype(np.int32)


@pytest.mark.parametrize("n,pockets", [(400_000, 1), (400_003, 40), (60_001, 7)])
def test_refused_while_ctas_start(built_lib, oracle_lib, n, pockets):
    import irregular_gb300 as irr
    edges = pocketed(n, pockets, n + pockets)
    both = np.concatenate([edges, edges[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    col = np.ascontiguousarray(both[:, 1], np.int32)
    assert oracle_lib.staged_layout(off, col) is None
    ref = oracle_lib.staged_layout(off, col, **WIDE)
    assert ref is not None
    pos = np.random.default_rng(1).random((n, 3)).astype(np.float32)

    def handle(**cfg):
        h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, **cfg))
        h.set_params(irr.minimd_params(6.25))
        h.set_edges(edges)
        h.set_nodes(pos, 12)
        return h

    for _ in range(4):
        h = handle()
        h.init()
        got = h.staged()
        for key in ("items", "slice_off", "words", "ids"):
            assert np.array_equal(got[key], ref[key]), key
        h.close()
        h = handle(layout=irr.IRR_LAYOUT_STAGED)
        with pytest.raises(irr.IrregularError) as ei:
            h.init()
        assert ei.value.status == irr.IRR_ERR_CAPACITY
        h.close()
