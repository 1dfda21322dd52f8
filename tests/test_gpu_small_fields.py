"""A field component much smaller than the others keeps its own precision, and
one that is zero stays zero."""
import numpy as np
import pytest

import oracle_lib as ol
import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu

AXES = {"x": 0, "y": 1, "z": 2}


def plasma(n, small, ratio, L, seed):
    """Electrons whose velocity along `small` is `ratio` times a thermal one."""
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3)) * 0.1
    u[:, AXES[small]] *= ratio
    g = np.sqrt(1 + (u * u).sum(1))[:, None]
    m = np.full(n, L * L / n)
    v = u / g
    return dict(x=rng.uniform(0, L, n), y=rng.uniform(0, L, n), P=u * m[:, None], v=v, vprev=v.copy(), q=-m, m=m)


def step(nx, ny, L, p, order, conserving):
    with up.Simulation(up.Config(nx=nx, ny=ny, Lx=L, Ly=L, dt=0.05, method="bdf%d" % order,
                                 charge_update="conserving" if conserving else "naive")) as sim:
        sim.set_particles(p["x"], p["y"], p["P"], p["v"], p["vprev"], p["q"], p["m"])
        sim.init_fields(False)
        sim.step(1, 0)
        return {a: sim.field("A" + a) for a in AXES}


# A after one step is linear in the current, (1/(c dt)^2 + k^2) A = mu0 J from
# A = 0: each component carries the relative rounding of its own current and
# transforms, the 1e-12 of its largest value that the other field tests allow.
@pytest.mark.parametrize("order,conserving", [(1, True), (2, False)])
@pytest.mark.parametrize("nx,ny", [(32, 64), (256, 128)])
@pytest.mark.parametrize("small", ["x", "y", "z"])
def test_small_component_against_oracle(nx, ny, small, order, conserving):
    L = 2 * np.pi / 0.3
    p = plasma(3000, small, 1e-8, L, nx + AXES[small])
    prob = ol.P2Problem(nx, ny, L, L, 0.05, order, conserving, n_steps=1)
    _, _, ref, _ = ol.simulate(ol.oracle().o2_simulate, prob, p)
    got = step(nx, ny, L, p, order, conserving)
    for a, k in AXES.items():
        r = ref[1 + k].reshape(got[a].shape)
        assert np.max(np.abs(got[a] - r)) < 1e-12 * np.max(np.abs(r)), a


@pytest.mark.parametrize("nx,ny", [(64, 64), (256, 256), (1024, 1024), (512, 2048)])
@pytest.mark.parametrize("zero", ["x", "y", "z"])
def test_zero_component_stays_zero(nx, ny, zero):
    L = 2 * np.pi / 0.3
    got = step(nx, ny, L, plasma(3000, zero, 0.0, L, nx), 1, True)
    for a in AXES:
        assert (np.max(np.abs(got[a])) == 0.0) == (a == zero), a
