"""Layouts made, dropped and made again by several threads at once (GPU), with
one pool between them: each handle's rows, layout and results are those of the
same handle made alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(n, per_row, span, seed):
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = rng.integers(0, n, i.size) if span is None else np.minimum(i + rng.integers(1, span + 1, i.size), n - 1)
    e = np.unique(np.stack([i, j], 1)[i != j], axis=0).astype(np.int32)
    return e, (rng.random((n, 3)) * 30).astype(np.float32)


def handle(irr, edges, pos, **cfg):
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MINIMD, reorder=0, **cfg))
    h.set_params(irr.minimd_params(6.25))
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    h.init()
    return h


def facts(irr, h):
    _, off, col = h.partition()
    got = [off, col]
    if h.info().layout == irr.IRR_LAYOUT_STAGED:
        got += [h.staged()[k] for k in ("items", "slice_off", "words", "ids")]
    h.step()
    return got + [h.get_result(elm_size=12).view(np.uint32)]


def in_threads(count, work):
    failed = []

    def run(k):
        try:
            work(k)
        except BaseException as e:  # noqa: BLE001 -- told to the test's own thread
            failed.append(f"thread {k}: {e!r}")

    ts = [threading.Thread(target=run, args=(k,)) for k in range(count)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed


def test_dropped_layouts(built_lib):
    """Random graphs (the staged layout is built, reuses too little and is
    dropped) beside banded ones (kept, then laid out again as slices, in a batch
    with a graph that does not fit it)."""
    import irregular_gb300 as irr
    inputs = [graph(30_000 + 7 * k, 8, None if k % 2 else 60, k) for k in range(6)]
    star = np.stack([np.zeros(3000, np.int32), np.arange(1, 3001, dtype=np.int32)], 1)
    star_pos = np.random.default_rng(9).random((3001, 3)).astype(np.float32)
    alone = []
    for e, pos in inputs:
        h = handle(irr, e, pos)
        alone.append(facts(irr, h))
        h.close()
    sliced = []
    for e, pos in inputs:
        h = handle(irr, e, pos, layout=irr.IRR_LAYOUT_SLICED)
        sliced.append(facts(irr, h))
        h.close()

    def work(k):
        e, pos = inputs[k]
        for _ in range(12):
            h = handle(irr, e, pos)
            for a, b in zip(facts(irr, h), alone[k]):
                assert np.array_equal(a, b)
            hub = handle(irr, star, star_pos)
            b = irr.Batch(0)
            b.add(h)
            b.add(hub)
            b.finalize()
            b.step()
            b.sync()
            assert h.info().layout != irr.IRR_LAYOUT_STAGED
            assert np.array_equal(h.get_result(elm_size=12).view(np.uint32), sliced[k][-1])
            for a, c in zip(facts(irr, h), sliced[k]):
                assert np.array_equal(a, c)
            b.close()
            hub.close()
            h.close()

    in_threads(len(inputs), work)


def test_setups_of_different_sizes(built_lib):
    """Items of few and of many entries: a set-up's launch takes the shared memory
    of its own largest item, whatever another thread's takes at that moment."""
    import irregular_gb300 as irr
    inputs = [graph(600 + 9 * k, 8 if k % 2 else 40, 60, k) for k in range(16)]
    alone = []
    for e, pos in inputs:
        h = handle(irr, e, pos)
        assert h.info().layout == irr.IRR_LAYOUT_STAGED
        alone.append(facts(irr, h))
        h.close()

    def work(k):
        e, pos = inputs[k]
        for _ in range(250):
            h = handle(irr, e, pos)
            h.step()
            got = h.get_result(elm_size=12).view(np.uint32)
            h.close()
            assert np.array_equal(got, alone[k][-1])

    in_threads(len(inputs), work)
