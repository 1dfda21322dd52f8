"""The closed-form local solve (2D, knot splitting, 2^19 particles and more)
and the private deposit windows where other tests do not reach them: particles
of different charge, quartic splines, warm starts, local solves that fail and
their log, orbits with more knots than the kernels hold.  The reference is the
Gauss-rule solve of the same plasma as half as many particles of twice the
charge and mass."""
import numpy as np
import pytest

import oracle_lib as ol
import unstaggered_pic_b200 as up
from unstaggered_pic_b200._native import UPIC_ERR

pytestmark = pytest.mark.gpu

L = 2 * np.pi / 0.3
N0 = 1e-3  # dilute: the local map is a contraction
HALF = 1 << 18
COL = {n: i for i, n in enumerate(up.FAILED_LOG_COLUMNS)}
# both solves end at 1e-11 of the velocity and the outer one at 1e-12 of the
# current, with a contraction of at most one half: 2 (1e-11 + 1e-12) / (1 - 1/2)
TOL_SOLVE = 1e-10


def relerr(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def plasma(order, two_species):
    x, v, q, m = ol.p3_particles(np.random.default_rng(order), 64, 64, 64, L, L, uth=(0.1, 0.2, 0.05), n0=N0)
    assert len(q) == HALF
    if two_species:  # a third of the particles: twice the charge, five times the mass, the other sign
        q[::3] *= -2.0
        m[::3] *= 5.0
    return x, v, q, m


def simulation(repeat, base, **kw):
    x, v, q, m = base
    r = lambda a: np.ascontiguousarray(np.repeat(a, repeat, axis=0))
    kw = {**dict(nx=64, ny=64, Lx=L, Ly=L, Lz=1.0, dt=0.05, n0=N0), **kw}
    sim = up.Simulation(up.ImplicitConfig(**kw))
    sim.set_particles(r(x[:, 0]), r(x[:, 1]), np.zeros((repeat * len(q), 3)), r(v), r(v), r(q) / repeat, r(m) / repeat)
    sim.init_fields()
    return sim


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("warm", [False, True])
def test_two_species_and_warm_starts(order, warm):
    base = plasma(order, True)
    res = []
    for repeat in (1, 2):
        with simulation(repeat, base, spline_order=order, local_warm_start=warm) as sim:
            sim.step_implicit(2)
            out = sim.get_particles()
            res.append((out["v"][::repeat], out["P"][::repeat] * repeat, np.stack([sim.field(f) for f in ("Jx", "Jy", "Jz")])))
    for a, b in zip(res[1], res[0]):
        assert relerr(a, b) < TOL_SOLVE


# The two logs hold the same failures; a residual of at least the tolerance
# 1e-3 |v| is the difference of velocities that agree to 1e-13 of |v|, so the
# logged values agree to 1e-9 of their column's largest.
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("case", ["slow", "light", "overflow"])
def test_failed_solves_and_their_log(order, case):
    x, v, q, m = plasma(order, False)
    some = np.array([3, 77, 4099, 200001, HALF - 1])
    want = "maximum_iterations"
    if case == "slow":       # uniform q/m; a tolerance relative to a velocity near zero
        v[some] *= 1e-6
    elif case == "light":    # their own q/m: one evaluation does not settle
        m[some] /= 3000.0
        q[some] /= 3.0
    else:                    # q/m that overflows
        m[some] = 1e-300
        want = "nonfinite_map"
    logs = []
    for repeat in (1, 2):
        with simulation(repeat, (x, v, q, m), spline_order=order, uniform_local_max_iter=1, uniform_local_rtol=1e-3) as sim:
            with pytest.raises(up.UpicError) as e:
                sim.step_implicit(1, diagnostics=False)
            assert UPIC_ERR[e.value.code] == "UPIC_ERR_LOCAL_PARTICLE"
            logs.append(sim.failed_particle_log())
    one, two = logs
    failed = set(one[:, COL["particle_index"]])
    # where its field happens to be weak, a light particle settles at once
    assert failed and (case == "light" or set(some) <= failed)
    assert np.all(one[:, COL["failure_reason"]] == up.FAILURE_REASONS.index(want))
    assert np.array_equal(two[:, COL["particle_index"]],
                          (2 * one[:, COL["particle_index"]][:, None] + (0, 1)).ravel())
    for name in ("failure_reason", "local_iterations", "assigned_substeps", "theta0", "theta1", "h"):
        assert np.array_equal(two[::2, COL[name]], one[:, COL[name]]), name
    if want == "maximum_iterations":
        for name in ("first_scaled_residual", "final_scaled_residual", "final_absolute_residual"):
            assert relerr(two[::2, COL[name]], one[:, COL[name]]) < 1e-9, name
        last = [COL[f"{k}_{c}"] for k in ("last_guess", "last_map") for c in "xyz"]
        assert relerr(two[::2][:, last], one[:, last]) < 1e-9
    assert np.array_equal(two[::2, 6:], two[1::2, 6:], equal_nan=True)


# 38 knots fit, 39 do not.
@pytest.mark.parametrize("cells,fits", [(38.2, True), (39.2, False)])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("axis", [0, 1])
def test_orbits_with_many_knots(axis, sign, cells, fits):
    """The closed-form solve (cells of size 1, orbits from the middle of a cell:
    quadratic splines have their knots at the half cells of the grid's offset)."""
    n0 = 1e-12
    rng = np.random.default_rng(5)
    n = 2 * HALF
    x = rng.uniform(-32, 32, (n, 2))
    v = rng.uniform(-0.01, 0.01, (n, 3))
    x[7] = (0.0, 0.0)  # knots of order 2 at half-integers: half a cell from the next either way
    v[7] = 0.0
    v[7, axis] = sign * cells / 50.0
    m = np.full(n, n0 * 64 * 64 / n)
    for cls in (up.ImplicitConfig, up.NonrelConfig):
        kw = dict(nx=64, ny=64, Lx=64.0, Ly=64.0, Lz=1.0, dt=50.0, n0=n0, guard=2)
        if cls is up.ImplicitConfig:
            kw.update(uniform_local_rtol=1e-9)
        with up.Simulation(cls(**kw)) as sim:
            sim.set_particles(x[:, 0], x[:, 1], np.zeros((n, 3)), v, v, -m, m)
            sim.init_fields()
            if fits:
                sim.step_implicit(1)
                out = sim.get_particles()
                d = np.array((out["x"][7], out["y"][7]))[axis] - sign * (cells - 64 * (cells > 32))
                assert abs(d) < 1e-3
                continue
            with pytest.raises(up.UpicError) as e:
                sim.step_implicit(1)
            if cls is up.ImplicitConfig:
                assert UPIC_ERR[e.value.code] == "UPIC_ERR_LOCAL_PARTICLE" and "knot" in str(e.value)
            else:
                assert UPIC_ERR[e.value.code] == "UPIC_ERR_TOO_LARGE"


# One step with private windows (default tile) and with one window per CTA (a
# tile of 32 cells takes more than the 75 KB that private ones may) on grids
# where the two differ.
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("nx,ny,n", [(32, 16, 1), (32, 16, 129), (32, 64, 1025), (64, 32, 20011)])
def test_private_windows_against_shared(nx, ny, n, order):
    x, v, q, m = ol.p3_particles(np.random.default_rng(n), n, 1, 1, L, L, uth=(0.1, 0.2, 0.05), n0=N0)
    res = []
    for tile in (0, 32):
        with simulation(1, (x, v, q, m), nx=nx, ny=ny, spline_order=order, tile=tile, guard=2) as sim:
            sim.step_implicit(1)
            out = sim.get_particles()
            res.append((out["v"], np.stack([sim.field(f) for f in ("Jx", "Jy", "Jz")])))
    for a, b in zip(*res):
        assert relerr(a, b) < TOL_SOLVE
