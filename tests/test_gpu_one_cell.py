"""Explicit steps with the conserving charge on grids one cell high or wide.
The momentum along that axis differs from the reference by 1e-8 (the imaginary
part of the continuity charge stays in the spectral histories; the expected
failures of test_gpu_windows.py), and the velocities with it.  Everything else
is held to the bounds of the other grids."""
import numpy as np
import pytest

import oracle_lib as ol
import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu

L = 2 * np.pi / 0.3


def relerr(a, b, scale=None):
    scale = np.max(np.abs(b)) if scale is None else scale
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b)))) / scale


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("tile", [0, 32])
@pytest.mark.parametrize("nx,ny", [(64, 1), (1, 64)])
def test_all_but_the_momentum_along_the_axis(nx, ny, tile, order):
    n = 3000
    rng = np.random.default_rng(nx)
    u = rng.normal(size=(n, 3)) * (0.1, 0.2, 0.05)
    v = u / np.sqrt(1 + (u * u).sum(1))[:, None]
    m = np.full(n, L * L / n)
    p = dict(x=rng.uniform(0, L, n), y=rng.uniform(0, L, n), P=u * m[:, None], v=v, vprev=v.copy(), q=-m, m=m)
    ref, _, rfields, _ = ol.simulate(ol.oracle().o2_simulate, ol.P2Problem(nx, ny, L, L, 0.05, order, True, n_steps=1), p)
    with up.Simulation(up.Config(nx=nx, ny=ny, Lx=L, Ly=L, dt=0.05, method="bdf%d" % order, tile=tile)) as sim:
        sim.set_particles(p["x"], p["y"], p["P"], p["v"], p["vprev"], p["q"], p["m"])
        sim.init_fields(False)
        sim.step(1, 0)
        out = sim.get_particles()
        fields = [sim.field(f) for f in ("phi", "Ax", "Ay", "Az", "rho", "Jx", "Jy", "Jz")]
    axis = 0 if nx == 1 else 1
    for k, rk in (("x", "x"), ("y", "y"), ("v_prev", "vprev")):
        assert relerr(out[k], ref[rk]) < 1e-13, k
    others = [c for c in range(3) if c != axis]
    assert relerr(out["P"][:, others], ref["P"][:, others], np.max(np.abs(ref["P"]))) < 1e-13
    assert relerr(out["P"], ref["P"]) < 1e-7 and relerr(out["v"], ref["v"]) < 1e-7
    scale = [np.max(np.abs(rfields[s])) for s in (slice(0, 1), slice(1, 4), slice(1, 4), slice(1, 4),
                                                  slice(4, 5), slice(5, 8), slice(5, 8), slice(5, 8))]
    for f in range(8):
        assert relerr(fields[f], rfields[f].reshape(fields[f].shape), scale[f]) < 1e-12, f
