"""A Picard iterate that overflows is an error: the deposit refuses its
velocities, and the push that is queued behind it ends whatever their size
(the knot searches themselves are checked on the CPU in test_orbit_knots.py)."""
import numpy as np
import pytest

import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [16, 1])
@pytest.mark.parametrize("order,quad", [(1, 8), (3, 8), (3, 2)])  # closed form; a rule of too few points: quadrature
@pytest.mark.parametrize("mass", [1e-20, 1e-40, 1e-300])
def test_overflowing_picard_iterate_is_an_error(mass, order, quad, ny):
    rng = np.random.default_rng(order)
    n = 200
    x, y = rng.uniform(-0.5, 0.5, (2, n))
    v = rng.uniform(-0.1, 0.1, (n, 3))
    cfg = up.NonrelConfig(nx=16, ny=ny, Lx=1.0, Ly=1.0, Lz=1.0, dt=0.05, spline_order=order, orbit_quad_order=quad)
    with up.Simulation(cfg) as sim:
        sim.set_particles(x, y, np.zeros((n, 3)), v, v, np.full(n, -1.0 / n), np.full(n, mass))
        sim.init_fields()
        with pytest.raises(up.UpicError, match="16 times the initial bound"):
            sim.step_implicit(1)
