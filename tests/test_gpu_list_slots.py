"""The one-pass neighbour list (slots per node) against the oracle's list, bit
for bit: cell counts around the fewest it takes, walls, open boundaries, nodes
in clusters that overflow their slots, positions on and outside the box."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(kind, n, side, rng):
    pos = (rng.random((n, 3)) * side).astype(np.float32)
    if kind == "cluster":  # a third of the nodes in one cell: more partners than slots
        pos[: n // 3] = (pos[: n // 3] * 0.05).astype(np.float32)
    elif kind == "plane":  # no extent on an axis
        pos[:, 2] = np.float32(0.5)
    elif kind == "walls":  # every coordinate at a wall
        pos = np.where(pos < side / 2, np.float32(0.0), np.nextafter(np.float32(side), np.float32(0))).astype(np.float32)
        pos += (rng.random((n, 3)) < 0.5) * np.float32(0.3) * np.where(pos < side / 2, 1, -1).astype(np.float32)
        pos = np.clip(pos, 0, np.nextafter(np.float32(side), np.float32(0))).astype(np.float32)
    elif kind == "outside":  # the cells then do not decide the images
        pos[::7] += np.float32(side * 0.01)
    pos[pos == np.float32(side)] = 0.0
    return pos


@pytest.mark.parametrize("kind", ["uniform", "cluster", "plane", "walls", "outside"])
@pytest.mark.parametrize("cells", [1, 2, 3, 4, 5, 6, 9])
@pytest.mark.parametrize("periodic", [True, False])
def test_list_equals_oracle(built_lib, oracle_lib, kind, cells, periodic):
    import irregular_gb300 as irr
    O = oracle_lib
    rc = 1.0
    side = float(np.float32(cells * rc * 1.01 + 0.05))
    n = 700 if kind != "walls" else 300
    pos = cloud(kind, n, side, np.random.default_rng(cells))
    cut2 = np.float32(rc * rc)
    ref = O.neighbor_half_list(pos, side if periodic else 0.0, cut2)
    got = irr.neighbor_build(pos, side if periodic else 0.0, float(cut2))
    assert got.count == len(ref)
    assert np.array_equal(got.to_host(), ref)


@pytest.mark.parametrize("n", [2, 31, 257, 5000])
@pytest.mark.parametrize("periodic", [True, False])
def test_sizes(built_lib, oracle_lib, n, periodic):
    import irregular_gb300 as irr
    O = oracle_lib
    side = float(np.float32(max(6.0, (n / 2.0) ** (1.0 / 3.0))))
    pos = cloud("uniform", n, side, np.random.default_rng(n))
    ref = O.neighbor_half_list(pos, side if periodic else 0.0, np.float32(1.0))
    got = irr.neighbor_build(pos, side if periodic else 0.0, 1.0)
    assert got.count == len(ref) and np.array_equal(got.to_host(), ref)
