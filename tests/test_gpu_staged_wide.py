"""The staged layout's wide limits (GPU): graphs whose 8 rows touch more nodes
than a narrow table holds.  AUTO takes them there; the layout equals the
oracle's restatement at those limits bit for bit, the results hold the other
layouts' bounds and repeat; an explicit IRR_LAYOUT_STAGED still refuses."""
import numpy as np
import pytest

from helpers import TOL_NORMWISE_F64, TOL_PERNODE_F64, normwise_error, random_box, scaled_error

pytestmark = pytest.mark.gpu

WIDE = dict(slices_per_item=8, tab_max=1008, stream_max=6400)


def system(O, n, neighbours, seed):
    rc = 2.5
    pos, side = random_box(n, neighbours / (4.0 / 3.0 * np.pi * rc ** 3), seed)
    return pos, float(side), rc, O.neighbor_half_list(pos, float(side), np.float32(rc * rc))


def handle(irr, pos, side, rc, edges, **cfg):
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MOLDYN, **cfg))
    h.set_params(irr.moldyn_params(side, rc))
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    h.init()
    return h


# sizes around whole blocks of 8 rows and a last block of one row
@pytest.mark.parametrize("n,neighbours", [(2000, 300), (2001, 260), (6007, 330), (40000, 248)])
def test_wide_layout_and_results(built_lib, oracle_lib, n, neighbours):
    import irregular_gb300 as irr
    O = oracle_lib
    pos, side, rc, edges = system(O, n, neighbours, 11)
    h = handle(irr, pos, side, rc, edges)
    assert h.info().layout == irr.IRR_LAYOUT_STAGED
    _, row_off, col = h.partition()
    ref, got = O.staged_layout(row_off, col), h.staged()
    if ref is None:  # the narrow limits do not hold this graph (they do at 2,001 nodes with 260)
        ref = O.staged_layout(row_off, col, **WIDE)
        with pytest.raises(irr.IrregularError) as ei:
            handle(irr, pos, side, rc, edges, layout=irr.IRR_LAYOUT_STAGED)
        assert ei.value.status == irr.IRR_ERR_CAPACITY
    else:
        assert (n, neighbours) == (2001, 260)
    for key in ("items", "slice_off", "words", "ids"):
        assert np.array_equal(got[key], ref[key]), key
    h.step()
    f = h.get_result(elm_size=12)
    f64, sabs = O.lj_reduce_f64(pos.astype(np.float64), edges, O.lj_param(rc * rc, side, True))
    assert normwise_error(f, f64) <= TOL_NORMWISE_F64
    assert scaled_error(f, f64, sabs) <= TOL_PERNODE_F64
    h.step()
    assert np.array_equal(h.get_result(elm_size=12).view(np.uint32), f.view(np.uint32))
    # a batch of such handles, and one mixed with narrow tables
    other = handle(irr, *system(O, 1500, 280, 12))
    small = handle(irr, *system(O, 1500, 30, 13))
    for instances in ([h, other], [h, small]):
        b = irr.Batch(0)
        for x in instances:
            b.add(x)
        b.finalize()
        b.step()
        b.sync()
        g = h.get_result(elm_size=12)
        assert scaled_error(g, f64, sabs) <= TOL_PERNODE_F64
        b.close()
    h.close()
