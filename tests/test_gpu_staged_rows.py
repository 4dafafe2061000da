"""The staged layout from rows in any order (GPU): the layout equals the
oracle's bit for bit and gives its rows back, for tables around the sizes at
which a row's bit map changes (256, 512) and an item is split (640), for rows
that name a node twice, and for edges in and out of idx0 order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def banded(n, band, per_row, repeats, seed):
    """Pairs (i, i + d), 0 < d <= band, the outermost among them; repeats: some
    of the pairs up to 5 times, and self edges."""
    rng = np.random.default_rng(seed)
    d = np.sort(rng.integers(1, band + 1, (n, per_row)), axis=1)
    d[:, 1:][d[:, 1:] == d[:, :-1]] = 0
    d[:, 0] = band
    i = np.repeat(np.arange(n), per_row)
    j = i + d.ravel()
    keep = (d.ravel() > 0) & (j < n)
    e = np.unique(np.stack([i[keep], j[keep]], 1), axis=0)
    if repeats:
        e = np.concatenate([e, e[::3], e[::17], e[::17], e[::17], np.stack([np.arange(0, n, 5)] * 2, 1)])
        e = e[np.argsort(e[:, 0], kind="stable")]
    return e.astype(np.int32)


@pytest.mark.parametrize("band", [1, 95, 96, 97, 223, 224, 225, 287, 288, 289, 400])
@pytest.mark.parametrize("repeats", [False, True])
def test_layout_and_rows(built_lib, oracle_lib, band, repeats):
    import irregular_gb300 as irr
    n = 1003
    rng = np.random.default_rng(band)
    edges = banded(n, band, min(band, 24), repeats, band)
    both = np.concatenate([edges, edges[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    ref = oracle_lib.staged_layout(off, both[:, 1].astype(np.int32))
    assert ref is not None
    for sorted_by_idx0 in (True, False):
        h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, layout=irr.IRR_LAYOUT_STAGED))
        h.set_params(irr.minimd_params(6.25))
        h.set_edges(edges if sorted_by_idx0 else np.ascontiguousarray(edges[rng.permutation(len(edges))]))
        h.set_nodes(rng.random((n, 3)).astype(np.float32), 12)
        h.init()
        got = h.staged()
        for key in ("items", "slice_off", "words", "ids"):
            assert np.array_equal(got[key], ref[key]), key
        for _ in range(2):  # made from the layout, then kept
            _, row_off, col = h.partition()
            assert np.array_equal(row_off, off) and np.array_equal(col, both[:, 1])
        h.close()


def test_sliced_after_staged(built_lib, oracle_lib):
    """A handle whose rows live in its staged layout, laid out again as slices
    (in a batch with a graph that does not fit the staged limits)."""
    import irregular_gb300 as irr
    n = 3001
    rng = np.random.default_rng(5)
    pos = rng.random((n, 3)).astype(np.float32) * 9
    star = np.stack([np.zeros(2000, np.int32), np.arange(1, 2001, dtype=np.int32)], 1)

    def handle(edges, **cfg):
        h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, **cfg))
        h.set_params(irr.minimd_params(6.25))
        h.set_edges(np.ascontiguousarray(edges))
        h.set_nodes(pos, 12)
        h.init()
        return h

    edges = banded(n, 200, 24, False, 1)
    want = handle(edges, layout=irr.IRR_LAYOUT_SLICED)
    want.step()
    h, hub = handle(edges), handle(star)
    assert h.info().layout == irr.IRR_LAYOUT_STAGED and hub.info().layout != irr.IRR_LAYOUT_STAGED
    b = irr.Batch(0)
    b.add(h)
    b.add(hub)
    b.finalize()
    b.step()
    b.sync()
    assert h.info().layout != irr.IRR_LAYOUT_STAGED
    a, c = h.get_result(elm_size=12), want.get_result(elm_size=12)
    assert np.array_equal(a.view(np.uint32), c.view(np.uint32))
    b.close()
    for x in (h, hub, want):
        x.close()
