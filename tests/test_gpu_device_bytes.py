"""irr_info.device_bytes of a staged handle counts the rows that
irr_get_partition makes from the layout and keeps (GPU)."""
import numpy as np
import pytest

from helpers import random_box

pytestmark = pytest.mark.gpu


def test_rows_kept_are_counted(built_lib, oracle_lib):
    import irregular_gb300 as irr
    pos, side = random_box(5000, 64 / (4.0 / 3.0 * np.pi * 2.5 ** 3), 8)
    edges = oracle_lib.neighbor_half_list(pos, float(side), np.float32(6.25))
    h = irr.Handle(irr.default_config(map_idx=irr.IRR_MAP_LJ_MOLDYN))
    h.set_params(irr.moldyn_params(float(side), 2.5))
    h.set_edges(edges)
    h.set_nodes(pos, 12)
    h.init()
    assert h.info().layout == irr.IRR_LAYOUT_STAGED
    before = h.info().device_bytes
    h.partition(with_entries=False)
    assert h.info().device_bytes == before
    for _ in range(2):
        h.partition()
        assert h.info().device_bytes == before + 4 * h.info().num_entries
    h.close()
