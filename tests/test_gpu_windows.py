"""Deposit windows, small sorts and the local solve's closed form at the sizes
where their launches change: particle counts around a round (256), a chunk
(1024, 2048) and a sort block, tiles whose windows are one per warp (the
default) and one per CTA (32 cells), grids that are no multiple of the tile and
one-cell axes, and particle counts around the closed form's first (2^19)."""
import numpy as np
import pytest

import oracle_lib as ol
import unstaggered_pic_b200 as up

pytestmark = pytest.mark.gpu

FIELDS = ("phi", "Ax", "Ay", "Az", "rho", "Jx", "Jy", "Jz")
L = 2 * np.pi / 0.3


def relerr(a, b, scale=None):
    a, b = np.asarray(a), np.asarray(b)
    if scale is None:
        scale = np.max(np.abs(b))
    d = float(np.max(np.abs(a - b))) if a.size else 0.0
    return d / scale if scale > 0 else d


def electrons(n, seed):
    """n electrons with velocities of both signs, all three components, q/m = -1
    and a total charge of -L^2."""
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(n, 3)) * (0.1, 0.2, 0.05)
    v = u / np.sqrt(1 + (u * u).sum(1))[:, None]
    m = np.full(n, L * L / n)
    return dict(x=rng.uniform(0, L, n), y=rng.uniform(0, L, n), P=u * m[:, None], v=v, vprev=v.copy(), q=-m, m=m)


def load(sim, p):
    sim.set_particles(p["x"], p["y"], p["P"], p["v"], p["vprev"], p["q"], p["m"])


# One step from the oracle: 1e-13 of the largest value per particle quantity,
# ten times that per field (the bounds of test_gpu_explicit.py).
@pytest.mark.parametrize("order,conserving", [(1, True), (2, False)])
@pytest.mark.parametrize("tile", [0, 32])
@pytest.mark.parametrize("nx,ny,n", [(16, 16, 1), (16, 16, 255), (16, 32, 256), (32, 16, 257), (32, 32, 1025),
                                     (64, 32, 2049), (32, 64, 70001), (64, 1, 3000), (1, 64, 3000)])
def test_explicit_step_by_count_and_tile(nx, ny, n, tile, order, conserving, request):
    if conserving and 1 in (nx, ny):
        # The wave number of a one-cell axis is -1 (the reference's numbering),
        # so the continuity charge has a spectrum that is not Hermitian.  The
        # reference drops its imaginary part with the real fields, the spectral
        # histories here keep it: the momentum along that axis differs by 1e-8.
        request.node.add_marker(pytest.mark.xfail(strict=True, reason="imaginary charge of a one-cell axis is kept"))
    p = electrons(n, 1000 * nx + n)
    prob = ol.P2Problem(nx, ny, L, L, 0.05, order, conserving, n_steps=1)
    ref, _, rfields, _ = ol.simulate(ol.oracle().o2_simulate, prob, p)
    with up.Simulation(up.Config(nx=nx, ny=ny, Lx=L, Ly=L, dt=0.05, method="bdf%d" % order, tile=tile,
                                 charge_update="conserving" if conserving else "naive")) as sim:
        load(sim, p)
        sim.init_fields(False)
        sim.step(1, 0)
        out = sim.get_particles()
        fields = [sim.field(f) for f in FIELDS]
    for k, rk in (("x", "x"), ("y", "y"), ("P", "P"), ("v", "v"), ("v_prev", "vprev")):
        assert relerr(out[k], ref[rk]) < 1e-13, k
    scale = [np.max(np.abs(rfields[s])) for s in (slice(0, 1), slice(1, 4), slice(1, 4), slice(1, 4),
                                                  slice(4, 5), slice(5, 8), slice(5, 8), slice(5, 8))]
    for f in range(8):
        assert relerr(fields[f], rfields[f], scale[f]) < 1e-12, FIELDS[f]


def test_particles_come_back_in_caller_order():
    """Whole values: ids carried as charges of distinct size, through several
    re-sorts; fp64 and mixed."""
    n = 5003
    p = electrons(n, 3)
    p["q"] = -np.arange(1, n + 1) / n * 1e-3
    p["m"] = np.abs(p["q"])
    p["P"] = p["v"] * (p["m"] / np.sqrt(1 - (p["v"] ** 2).sum(1)))[:, None]
    for precision in ("fp64", "mixed"):
        with up.Simulation(up.Config(nx=32, ny=32, Lx=L, Ly=L, dt=0.01, sort_interval=1, precision=precision)) as sim:
            load(sim, p)
            sim.init_fields(False)
            sim.step(3, 0)
            out = sim.get_particles()
        # within the free flight of three steps, which no two ids share
        tol = 1e-2 if precision == "fp64" else 2e-2
        d = out["x"] - (p["x"] + 0.03 * p["v"][:, 0])
        assert np.max(np.abs(d - L * np.round(d / L))) < tol
        d = out["y"] - (p["y"] + 0.03 * p["v"][:, 1])
        assert np.max(np.abs(d - L * np.round(d / L))) < tol


@pytest.mark.parametrize("nsteps", [63, 64, 65, 130])
def test_rows_of_one_call_are_those_of_single_steps(nsteps):
    """More rows than are in flight at a time, bit for bit."""
    p = electrons(3000, 9)
    rows = []
    for split in (False, True):
        with up.Simulation(up.Config(nx=16, ny=16, Lx=L, Ly=L, dt=0.05)) as sim:
            load(sim, p)
            sim.init_fields(False)
            rows.append(np.vstack([sim.step(1, 1) for _ in range(nsteps)]) if split else sim.step(nsteps, 1))
    assert np.array_equal(rows[0], rows[1])


# A dilute plasma: the field of one particle alone leaves the solve a contraction.
N0 = 1e-3


def implicit(n_repeat, base, **kw):
    """One step of `base` with every particle as n_repeat equal parts."""
    x, v, q, m = base
    cfg = up.ImplicitConfig(Lx=L, Ly=L, Lz=1.0, dt=0.05, n0=N0, **kw)
    with up.Simulation(cfg) as sim:
        r = lambda a: np.ascontiguousarray(np.repeat(a, n_repeat, axis=0))
        sim.set_particles(r(x[:, 0]), r(x[:, 1]), np.zeros((n_repeat * len(q), 3)), r(v), r(v), r(q) / n_repeat,
                          r(m) / n_repeat)
        sim.init_fields()
        sim.step_implicit(1)
        out = sim.get_particles()
        return out["v"][::n_repeat], np.stack([sim.field(f) for f in ("Jx", "Jy", "Jz")])


# The outer solve ends at 1e-12 of the current and the local ones at 1e-11 of
# the velocity; with a contraction of at most one half two runs that round
# differently end within 2 (1e-11 + 1e-12) / (1 - 1/2) < 1e-10.
TOL_SOLVE = 1e-10


@pytest.mark.parametrize("order", [1, 2, 3])
def test_closed_form_solve_matches_gauss_rule(order):
    """2^18 particles take the Gauss rule; the same plasma as 2^19 halves takes
    the closed form."""
    base = ol.p3_particles(np.random.default_rng(order), 64, 64, 64, L, L, uth=(0.1, 0.2, 0.05), n0=N0)
    assert len(base[2]) == 1 << 18
    kw = dict(nx=64, ny=64, spline_order=order)
    va, ja = implicit(1, base, **kw)
    vb, jb = implicit(2, base, **kw)
    assert relerr(vb, va) < TOL_SOLVE
    assert relerr(jb, ja) < TOL_SOLVE


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("nx,ny,n", [(16, 16, 1), (16, 16, 129), (32, 16, 1025), (32, 64, 20011), (64, 1, 4099)])
def test_implicit_deposit_by_count_and_tile(nx, ny, n, order):
    """Windows per warp (default tile) against one per CTA (32-cell tile)."""
    x, v, q, m = ol.p3_particles(np.random.default_rng(n), n, 1, 1, L, L, uth=(0.1, 0.2, 0.05), n0=N0)
    res = [implicit(1, (x, v, q, m), nx=nx, ny=ny, spline_order=order, tile=t) for t in (0, 32)]
    assert relerr(res[1][0], res[0][0]) < TOL_SOLVE
    assert relerr(res[1][1], res[0][1]) < TOL_SOLVE
