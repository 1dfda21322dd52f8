"""Deposits whose large parts cancel: what is left is as exact as it would be
without them, however many particles of a tile a warp sums (a plain FP64
running sum would keep an ulp of the large part)."""
import numpy as np
import pytest

import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu


# Particles on a node (weights 1/8, 3/4, 1/8), cell size 1 and velocities and
# charges that are powers of two times small integers: every product and the
# sum are exact, and the accumulators' resolution (2^-91 of a bound of 2^50)
# holds them, so the result is exact.  Every warp gets batches of both signs.
@pytest.mark.parametrize("charge", ["naive", "conserving"])
@pytest.mark.parametrize("nx,ny", [(16, 16), (32, 64)])
def test_explicit_sums_are_exact(nx, ny, charge):
    big, n = 2.0 ** 40, 256
    small = 2.0 ** -20 * (1 + np.arange(n) % 7)
    q = np.concatenate([np.full(n, big), small, np.full(n, -big)])
    v = np.tile((0.5, -0.25, 0.125), (3 * n, 1))
    m = np.full(3 * n, big)
    P = v * m[:, None] / np.sqrt(1 - (v * v).sum(1))[:, None]
    x, y = 5.0, 6.0
    with up.Simulation(up.Config(nx=nx, ny=ny, Lx=float(nx), Ly=float(ny), dt=4.0, charge_update=charge)) as sim:
        sim.set_particles(np.full(3 * n, x), np.full(3 * n, y), P, v, v, q, m)
        sim.init_fields(False)
        # at the start, and one free flight of (2, -1) cells later
        for k in range(2):
            w = np.zeros((nx, ny))
            w[np.ix_([4 + 2 * k, 5 + 2 * k, 6 + 2 * k], [5 - k, 6 - k, 7 - k])] = np.outer((0.125, 0.75, 0.125),
                                                                                          (0.125, 0.75, 0.125))
            for c, f in enumerate(("Jx", "Jy", "Jz")):
                assert np.array_equal(sim.field(f), small.sum() * v[0, c] * w), (k, f)
            if k == 0:
                sim.step(1, 0)


# Particles too heavy to be moved (q/m = 1e-30), so equal orbits, in blocks of
# 128 with charges +big, 1, -big: runs of equal magnitude and opposite sign
# cancel exactly, and the current is that of the unit charges alone.  What is
# left is the accumulators' resolution, 2^-91 of the bound 256000 big v = 2^60,
# in at most 12000 sums of 32 particles each: 1e-10 of the current of 128000
# unit charges.  A running FP64 sum loses up to 2^-6 per warp, 1e-6 and more.
@pytest.mark.parametrize("method", ["implicit", "nonrel"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_orbit_sums_keep_small_charges(order, method):
    blocks, big = 1000, 2.0 ** 42
    one = np.repeat((big, 1.0, -big), 128)
    q = np.tile(one, blocks)
    kw = dict(nx=32, ny=32, Lx=32.0, Ly=32.0, Lz=1.0, dt=0.5, spline_order=order, orbit_quad_order=8)
    v1 = np.array((0.4, -0.3, 0.2))

    def current(q):
        n = len(q)
        v = np.tile(v1, (n, 1))
        cfg = (up.ImplicitConfig(split_orbit_at_knots=True, **kw) if method == "implicit" else up.NonrelConfig(**kw))
        with up.Simulation(cfg) as sim:
            sim.set_particles(np.full(n, 3.3), np.full(n, -2.6), np.zeros((n, 3)), v, v, q, 1e30 * np.abs(q))
            sim.init_fields()
            sim.step_implicit(1)
            return np.stack([sim.field(f) for f in ("Jx", "Jy", "Jz")])

    want = current(q[q == 1.0])
    got = current(q)
    assert np.max(np.abs(want)) > 1000.0
    assert np.max(np.abs(got - want)) < 1e-9 * np.max(np.abs(want))
