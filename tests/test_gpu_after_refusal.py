"""A context that cannot be created (a deposit window larger than an SM's shared
memory) leaves nothing behind: the next one runs as if it were the first."""
import numpy as np
import pytest

import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu


def run(method):
    n = 5000
    rng = np.random.default_rng(3)
    v = rng.uniform(-0.1, 0.1, (n, 3))
    m = np.full(n, 25.0 / n)
    x, y = rng.uniform(0, 5, (2, n))
    if method in ("bdf1", "mixed"):
        cfg = up.Config(nx=32, ny=32, Lx=5.0, Ly=5.0, dt=0.02, precision="mixed" if method == "mixed" else "fp64")
        P = v * (m / np.sqrt(1 - (v * v).sum(1)))[:, None]
    else:
        cls = up.ImplicitConfig if method == "cn_orbit" else up.NonrelConfig
        cfg, P = cls(nx=32, ny=32, Lx=5.0, Ly=5.0, Lz=1.0, dt=0.02), np.zeros((n, 3))
        x, y = x - 2.5, y - 2.5
    with up.Simulation(cfg) as sim:
        sim.set_particles(x, y, P, v, v, -m, m)
        sim.init_fields()
        sim.step(2) if method in ("bdf1", "mixed") else sim.step_implicit(2)
        return sim.get_particles()["v"].copy()


@pytest.mark.parametrize("refused", [dict(tile=32), dict(tile=64, charge_update="naive"), dict(tile=64, implicit=True)])
@pytest.mark.parametrize("method", ["bdf1", "mixed", "cn_orbit", "cn_orbit_nonrel"])
def test_run_after_a_refused_creation(method, refused):
    want = run(method)
    kw = dict(nx=256, ny=256, Lx=5.0, Ly=5.0, **{k: v for k, v in refused.items() if k != "implicit"})
    cfg = up.ImplicitConfig(Lz=1.0, **kw) if refused.get("implicit") else up.Config(**kw)
    with pytest.raises(up.UpicError):
        up.Simulation(cfg)
    assert np.array_equal(run(method), want)
