"""AUTO's choice by reuse (GPU): the staged layout, to the narrow limits or else
to the wide ones, where its tables hold at most a third as many ids as the rows
hold entries (as the oracle lays them out), else slices or CSR; on both sides of
the line, whether the narrow limits hold the graph or not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDE = dict(slices_per_item=8, tab_max=1008, stream_max=6400)


def graph(n, per_row, span, seed):
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = i + rng.integers(1, span + 1, i.size)
    e = np.unique(np.stack([i, j], 1)[j < n], axis=0).astype(np.int32)
    both = np.concatenate([e, e[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    return e, off, np.ascontiguousarray(both[:, 1])


# (rows, edges per row, how far their partners are): reuse 0.9 to 11
GRAPHS = [(5003, 1, 2), (5003, 2, 2), (5003, 2, 4), (5003, 2, 14), (5003, 2, 18), (5003, 2, 22), (5003, 4, 60),
          (5003, 4, 100), (5003, 4, 140), (5003, 4, 3000), (5003, 20, 400), (5003, 20, 600), (5003, 60, 700),
          (5003, 60, 900), (5003, 60, 4000), (5003, 100, 440), (5003, 100, 2000), (40001, 60, 30000)]


def test_choice(built_lib, oracle_lib):
    import irregular_gb300 as irr
    seen = set()
    for k, (n, per_row, span) in enumerate(GRAPHS):
        edges, off, col = graph(n, per_row, span, k)
        kind, ref = "narrow", oracle_lib.staged_layout(off, col)
        if ref is None:
            kind, ref = "wide", oracle_lib.staged_layout(off, col, **WIDE)
        if ref is None:
            kind = "none"
        pays = ref is not None and len(col) >= 3 * len(ref["ids"])
        seen.add((kind, pays))
        h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0))
        h.set_params(irr.minimd_params(6.25))
        h.set_edges(edges)
        h.set_nodes(np.random.default_rng(k).random((n, 3)).astype(np.float32), 12)
        h.init()
        assert (h.info().layout == irr.IRR_LAYOUT_STAGED) == pays, (n, per_row, span, kind)
        if pays:
            got = h.staged()
            for key in ("items", "slice_off", "words", "ids"):
                assert np.array_equal(got[key], ref[key]), key
        _, row_off, rows = h.partition()
        assert np.array_equal(row_off, off) and np.array_equal(rows, col)
        h.close()
    assert seen == {("narrow", True), ("narrow", False), ("wide", True), ("wide", False), ("none", False)}
