"""The MD integrator's integer-unit conversions and box wrap (GPU), bit for bit
against the rules in exact arithmetic: float copies of positions that lie on and
around the ties of the rounding, half kicks by forces (zero among them), and
atoms that cross the box's faces, by a rounding error or by more than a box."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # one rounding, to nearest even


def wrap(x, side):
    if x >= side:
        x = x - side if x < 2 * side else x - side * np.floor(x / side)
    elif x < 0:
        x = x + side if x >= -side else x - side * np.floor(x / side)
    if x >= side:
        x -= side
    return 0.0 if x < 0 else x


def test_float_copies_and_half_kicks(built_lib):
    import irregular_gb300 as irr
    rng = np.random.default_rng(2)
    m, a = 8, 1.7
    pos = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3) * a
    pos = pos + rng.uniform(0.05, 0.35, pos.shape)
    q = pos.astype(np.float32)
    half = (np.nextafter(q, np.float32(np.inf)).astype(np.float64) - q) / 2
    off = rng.integers(-1, 2, pos.shape) * np.spacing(q + half)  # a double's step below a tie, on it, above
    pos = q + half * rng.integers(0, 2, pos.shape) + off * rng.integers(0, 2, pos.shape)
    pos[0] = (0.0, 2.0 ** -30, 1e-30)  # zero takes the instruction
    dt = 1e-14  # too short to move what a float copy shows
    md = irr.MD(pos, np.zeros_like(pos), m * a, dt=dt)
    f = md.forces()
    md.run(1)
    x, v = md.state()
    assert np.array_equal(md.forces().view(np.uint64), f.view(np.uint64))
    hk = 0.5 * dt * 48.0
    for g, got, before, after in zip((f / 48.0).ravel()[:600], v.ravel()[:600], pos.ravel(), x.ravel()):
        v1 = fma(hk, g, 0.0)
        assert got == fma(hk, g, v1)
        assert after == wrap(fma(dt, v1, before), m * a)
    md.close()


def test_box_wrap(built_lib):
    import irregular_gb300 as irr
    side, dt = 400.0, 0.5
    up = np.nextafter
    ends = [side, up(side, 0), up(side, 1e9), up(side * (1 - 2.0 ** -21), 0), side * (1 - 2.0 ** -20), 0.0, -0.0, -1e-300,
            -2.0 ** -60, up(0, -1), -1.0, -side, up(-side, 0), -1.5 * side, 2 * side, up(2 * side, 0), 2.5 * side,
            0.25, 399.0, 400.25, 1e-40]
    # atoms too far apart for forces, at rest on two axes
    x0 = np.stack(np.meshgrid(*(np.arange(4),) * 3, indexing="ij"), -1).reshape(-1, 3) * 100.0 + 50.0
    vel = np.zeros_like(x0)
    want = x0.copy()

    for k, end in enumerate(ends):
        c = k % 3
        x0[k, c] = 0.0 if abs(end) < 0.2 else x0[k, c]
        vel[k, c] = (end - x0[k, c]) / dt
        want[k, c] = wrap(fma(dt, vel[k, c], x0[k, c]), side)
    md = irr.MD(x0, vel, side, dt=dt, rebuild_every=1000)
    assert not md.forces().any()
    md.run(1)
    x, v = md.state()
    assert np.array_equal(v, vel)
    assert np.array_equal(x, want)
    md.run(1)  # the fused kick and drift
    x2, _ = md.state()
    assert np.array_equal(x2, np.vectorize(lambda p, u: wrap(fma(dt, u, p), side))(want, vel))
    md.close()
