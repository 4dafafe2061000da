"""The plain executor's run-summed atomics (GPU): lists whose idx0 runs end
inside a warp, span warps, or do not repeat, at sizes around a warp's 32 edges,
against the FP64 oracle within the tolerances of the other executors."""
import numpy as np
import pytest

from helpers import TOL_NORMWISE_F64, TOL_PERNODE_F64, normwise_error, random_box, scaled_error

pytestmark = pytest.mark.gpu

RHO64 = 64.0 / (4.0 / 3.0 * np.pi * 2.5 ** 3)


def edge_list(O, pos, side, order, rng):
    edges = O.neighbor_half_list(pos, float(side), np.float32(6.25))
    if order == "shuffled":  # hardly ever a repeated idx0 within a warp
        edges = edges[rng.permutation(len(edges))]
    elif order == "star":  # one run over many warps
        edges = np.stack([np.full(len(pos) - 1, 7), np.delete(np.arange(len(pos)), 7)], 1).astype(np.int32)
    elif order == "pairs":  # runs of two, one of them cut by the warp's end
        edges = np.roll(edges[rng.permutation(len(edges))].repeat(2, axis=0), 1, axis=0)
    return np.ascontiguousarray(edges)


@pytest.mark.parametrize("order", ["sorted", "shuffled", "star", "pairs"])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 64, 255, 257, 5000, None])
@pytest.mark.parametrize("periodic", [True, False])
def test_runs_against_fp64(built_lib, oracle_lib, order, count, periodic):
    import irregular_gb300 as irr
    O = oracle_lib
    pos, side = random_box(1500, RHO64, 77)
    edges = edge_list(O, pos, side, order, np.random.default_rng(5))[:count]
    p = O.lj_param(6.25, float(side) if periodic else 0.0, periodic)
    f64, sabs = O.lj_reduce_f64(pos.astype(np.float64), edges, p)
    h = irr.Handle(irr.default_config(exec=irr.IRR_EXEC_PLAIN,
                                      map_idx=irr.IRR_MAP_LJ_MOLDYN if periodic else irr.IRR_MAP_LJ_MINIMD))
    h.set_params(irr.moldyn_params(float(side), 2.5) if periodic else irr.minimd_params(6.25))
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    for _ in range(2):  # the second step clears the first one's results
        h.step()
        f = h.get_result(elm_size=12)
        if np.abs(f64).max() > 0:
            assert normwise_error(f, f64) <= TOL_NORMWISE_F64
        assert scaled_error(f, f64, sabs) <= TOL_PERNODE_F64
        assert not f[sabs.max(axis=1) == 0 if sabs.ndim > 1 else sabs == 0].any()
    h.close()
