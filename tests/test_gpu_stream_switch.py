"""irr_set_stream with steps in flight on the old stream (GPU): what the handle
then frees, to hold a longer list, more records or wider results, is not handed
out again before those steps have ended."""
import numpy as np
import pytest

from helpers import TOL_NORMWISE_F64, normwise_error, random_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["plain", "partitioned"])
def test_growing_after_a_switch(built_lib, oracle_lib, mode):
    torch = pytest.importorskip("torch")
    import irregular_gb300 as irr
    O = oracle_lib
    rc, n = 2.5, 20_000
    pos, side = random_box(n, 200 / (4.0 / 3.0 * np.pi * rc ** 3), 5)
    edges = O.neighbor_half_list(pos, float(side), np.float32(rc * rc))
    f64, _ = O.lj_reduce_f64(pos.astype(np.float64), edges, O.lj_param(rc * rc, float(side), True))

    def handle(e, p):
        h = irr.Handle(irr.default_config(
            map_idx=irr.IRR_MAP_LJ_MOLDYN,
            exec=irr.IRR_EXEC_PLAIN if mode == "plain" else irr.IRR_EXEC_PARTITIONED))
        h.set_params(irr.moldyn_params(float(side), rc))
        h.set_edges(e)
        h.set_nodes(p, 12)
        return h

    old, new = torch.cuda.Stream(), torch.cuda.Stream()
    zero = np.zeros_like(edges)  # of the old list's size: valid ids, no force
    for _ in range(3):
        h = handle(edges, pos)
        h.set_stream(old.cuda_stream)
        h.init()
        out = torch.zeros((n, 4), device="cuda")
        torch.cuda.synchronize()
        for _ in range(400):
            h.step()
        h.get_result_device(out, 16)
        h.set_stream(new.cuda_stream)
        h.set_edges(np.concatenate([edges, edges[:1000]]))  # a longer list: the old one's block is free
        other = handle(zero, pos[::-1].copy())  # and taken
        other.init()
        torch.cuda.synchronize()
        got = out[:, :3].cpu().numpy()
        assert normwise_error(got, f64) <= TOL_NORMWISE_F64
        h.init()
        h.step()
        assert np.isfinite(h.get_result(elm_size=24)).all()
        other.close()
        h.close()
