"""The MD rebuild's rows (GPU) against the oracle's list, with 8 lanes per node
and with one (40,000 nodes and below, above), for cells of few and of many
nodes: the pair count, and the forces of the rows."""
import numpy as np
import pytest

from helpers import TOL_PERNODE_F64, random_box, scaled_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,neighbours", [(1500, 40), (1501, 250), (5003, 100), (39999, 60), (40000, 60), (40001, 60),
                                          (40005, 200)])
def test_pairs_and_forces(built_lib, oracle_lib, n, neighbours):
    import irregular_gb300 as irr
    O = oracle_lib
    pos, side = random_box(n, neighbours / (4.0 / 3.0 * np.pi * 2.8 ** 3), n)
    side = float(side)
    md = irr.MD(pos.astype(np.float64), np.zeros((n, 3)), side, dt=1e-9, rebuild_every=2)
    for steps in (0, 2):  # the first build (two searches), a rebuild (one, into slots)
        md.run(steps)
        q = md.state()[0].astype(np.float32)
        edges = O.neighbor_half_list(q, float(np.float32(side)), np.float32(2.8 ** 2))
        assert md.info().num_edges == len(edges) > 0
        f64, sabs = O.lj_reduce_f64(q.astype(np.float64), edges, O.lj_param(2.5 ** 2, side, True))
        assert scaled_error(md.forces(), 48.0 * f64, 48.0 * sabs) <= TOL_PERNODE_F64
    md.close()
