"""Performance cases: the particle-in-cell steps a user of this framework runs.

Every case is a run in progress: `prepare` creates the simulation, loads a
seeded plasma and starts its fields; one pass (`run`) advances it by a number
of steps and reads the state back into buffers the caller keeps, as a driver
does between two dumps.  The plasmas are the ones of bench.py: Weibel
bi-Maxwellians (u_th 0.02 / 0.2 c), a bulk with a 0.5 c beam of another
charge, and counter-drifting 1D-2V beams.
"""
import math

import numpy as np
import torch

import unstaggered_pic_b200 as up

L512 = 2 * math.pi / 0.3                 # box edge of the 512-cell workloads
H = L512 / 512                           # their cell size
FIELDS = ["phi", "Ax", "Ay", "Az", "rho", "Jx", "Jy", "Jz"]
# the manuscript deck's solver settings in 2D
DECK = dict(Lz=1.0, kappa=1.0, sigma1=1.0, sigma2=1.0, n0=1.0, orbit_quad_order=8, split_orbit_at_knots=True,
            nyquist_projection=True, nonlinear_solver="anderson_quasi_newton", nonlinear_rtol=1e-11,
            nonlinear_atol=1e-13, nonlinear_max_iter=80, anderson_memory=4, anderson_start=2, anderson_damping=0.5,
            anderson_regularization=1e-12, anderson_growth_limit=1.2, uniform_local_rtol=1e-12,
            uniform_local_atol=1e-14, uniform_local_max_iter=64, uniform_local_damping=1.0)
# runs of an ensemble: grid by turns, particle counts spread between the case's limits
ENSEMBLE_GRIDS = [(16, 8), (16, 16), (32, 16), (32, 32)]
ENSEMBLE_NX_1D = [128, 256, 512, 1024]


def explicit(name, nx, ny, particles, method="bdf1", charge="conserving", precision="fp64", beam=False, steps=50,
             stride=10):
    return {"name": name, "kind": "explicit", "nx": nx, "ny": ny, "particles": particles, "method": method,
            "charge": charge, "precision": precision, "beam": beam, "steps": steps, "stride": stride}


def implicit(name, nx, ny, particles, order, dt, steps, predictor="previous", two_stream=False):
    return {"name": name, "kind": "implicit", "nx": nx, "ny": ny, "particles": particles, "order": order, "dt": dt,
            "steps": steps, "predictor": predictor, "two_stream": two_stream}


def nonrel(name, nx, ny, particles, order, steps):
    return {"name": name, "kind": "nonrel", "nx": nx, "ny": ny, "particles": particles, "order": order, "dt": 0.05,
            "steps": steps}


def ensemble(name, method, runs, least, most, steps):
    return {"name": name, "kind": "ensemble", "method": method, "runs": runs, "least": least, "most": most,
            "steps": steps}


def listed():
    return [
        # the smallest explicit run, diagnostics every step (the default): launches and latency count
        explicit("explicit_32x32_16k", 32, 32, 16 * 1024, stride=1),
        # the CPU-runnable configuration of the reference's Weibel decks, second-order BDF
        explicit("explicit_64x64_262k_bdf2", 64, 64, 64 * 4096, method="bdf2", stride=1),
        # an oblong grid, two populations of different charge, naive charge update, a ragged count
        explicit("explicit_256x128_1m_beam", 256, 128, 999_983, charge="naive", beam=True),
        # a production run: the headline grid at 64 electrons per cell
        explicit("explicit_512x512_17m", 512, 512, 64 * 512 * 512),
        # a large grid with few particles per cell in the mixed-precision form
        explicit("mixed_1024x1024_8m", 1024, 1024, 8 * 1024 * 1024, precision="mixed"),
        # a parameter scan of small explicit runs advanced together
        ensemble("ensemble_32_explicit", "bdf1", 32, 10_000, 100_000, 120),
        # the energy-conserving implicit step where a step is a few small kernels
        implicit("implicit_64x64_66k", 64, 64, 16 * 4096, 2, 0.05, 4),
        # the same method on the headline grid
        implicit("implicit_512x512_4m", 512, 512, 16 * 512 * 512, 2, 0.05, 2),
        # cubic splines in 2D, ragged count, extrapolated first guess
        implicit("implicit_256x256_1m_cubic", 256, 256, 1_000_003, 3, 0.05, 2, predictor="extrapolated"),
        # a 1D-2V two-stream run with cubic splines
        implicit("implicit_512x1_150k_cubic", 512, 1, 150_001, 3, 0.1, 4, two_stream=True),
        # a parameter scan of 1D-2V two-stream runs advanced together
        ensemble("ensemble_16_implicit_1d", "cn_orbit", 16, 10_000, 100_000, 2),
        # the non-relativistic Picard method, quadratic splines
        nonrel("nonrel_128x128_524k", 128, 128, 32 * 128 * 128, 2, 3),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["explicit", "explicit", "mixed", "implicit", "implicit_1d", "nonrel", "ensemble"])
    if kind in ("explicit", "mixed"):
        nx, ny = 2 ** rng.randint(5, 9), 2 ** rng.randint(5, 9)
        n = log_int(4 * nx * ny, min(96 * nx * ny, 1.6e7))
        c = explicit("", nx, ny, n, rng.choice(["bdf1", "bdf2"]), rng.choice(["conserving", "naive"]),
                     "fp64" if kind == "explicit" else "mixed", rng.random() < 0.3,
                     rng.choice([20, 30, 40]), rng.choice([1, 5, 10]))
    elif kind == "implicit":
        nx, ny = 2 ** rng.randint(4, 8), 2 ** rng.randint(4, 8)
        n = log_int(8 * nx * ny, min(64 * nx * ny, 1.0e6))
        c = implicit("", nx, ny, n, rng.choice([1, 2, 2, 3]), rng.choice([0.05, 0.1]), rng.choice([1, 2]),
                     rng.choice(["previous", "extrapolated"]))
    elif kind == "implicit_1d":
        nx = 2 ** rng.randint(7, 10)
        c = implicit("", nx, 1, log_int(1e4, 4e5), rng.choice([2, 3, 3]), 0.1, rng.choice([2, 3]),
                     rng.choice(["previous", "extrapolated"]), True)
    elif kind == "nonrel":
        nx, ny = 2 ** rng.randint(4, 8), 2 ** rng.randint(0, 8)
        n = log_int(8 * nx * ny + 4096, min(128 * nx * ny + 8192, 1.0e6))
        c = nonrel("", nx, ny, n, rng.choice([1, 2, 2, 3]), rng.choice([1, 2]))
    else:
        method = rng.choice(["bdf1", "bdf1", "cn_orbit"])
        runs = rng.randint(4, 24) if method == "bdf1" else rng.randint(3, 12)
        c = ensemble("", method, runs, log_int(5e3, 2e4), log_int(4e4, 9e4), 80 if method == "bdf1" else 1)
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------
def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def box(c):
    """Cell size of the 512-cell workloads; a 64-cell run of the decks has a
    full-size box, so small grids take coarser cells."""
    h = H * max(1.0, 512 / max(c["nx"], c["ny"], 64)) ** 0.5
    return c["nx"] * h, (c["ny"] * h if c["ny"] > 1 else 1.0)


def plasma(c, seed):
    """x, y in [0, L), u = gamma v (or v), q, m: float64 tensors."""
    g = torch.Generator(device=device()).manual_seed(1_000_003 * (int(seed) % 1_000_000_007) + 17)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=device(), dtype=torch.float64)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=device(), dtype=torch.float64)

    n, nx, ny = c["particles"], c["nx"], c["ny"]
    Lx, Ly = box(c)
    if c.get("two_stream"):
        v0 = c["v0"]
        Lx = 2 * math.pi * v0 / 0.6 * 4  # four wavelengths of the fastest-growing cold mode
        u = torch.zeros(n, 3, device=device(), dtype=torch.float64)
        u[: n // 2, 0], u[n // 2:, 0] = v0, -v0
        u[:, :2] += 0.01 * normal(n, 2)
        q = torch.full((n,), -Lx / n, device=device(), dtype=torch.float64)
        return Lx, Ly, Lx * rand(n), 0.5 + torch.zeros_like(q), u, q, -q
    # stratified over the cells, which a particle's index runs through in order
    cell = torch.div(torch.arange(n, device=device()) * (nx * ny), n, rounding_mode="floor")
    i, j = torch.div(cell, ny, rounding_mode="floor"), cell % ny
    x, y = (i + rand(n)) * (Lx / nx), (j + rand(n)) * (Ly / ny)
    spread = torch.tensor([0.02, 0.2, 0.0 if c["kind"] != "nonrel" else 0.05], device=device(), dtype=torch.float64)
    u = normal(n, 3) * spread
    w = torch.full((n,), Lx * Ly / n, device=device(), dtype=torch.float64)
    if c.get("beam"):
        late = rand(n) < 6 / 64
        u[late, 1] += 0.5
        w[late] *= 1.0625
    return Lx, Ly, x, y, u, -w, w.clone()


def config(c, Lx, Ly):
    if c["kind"] == "explicit":
        return up.Config(nx=c["nx"], ny=c["ny"], Lx=Lx, Ly=Ly, dt=0.05, method=c["method"], charge_update=c["charge"],
                         precision=c["precision"])
    if c["kind"] == "nonrel":
        return up.NonrelConfig(nx=c["nx"], ny=c["ny"], Lx=Lx, Ly=Ly, Lz=1.0, dt=c["dt"], spline_order=c["order"],
                               orbit_quad_order=8)
    return up.ImplicitConfig(nx=c["nx"], ny=c["ny"], Lx=Lx, Ly=Ly, dt=c["dt"], spline_order=c["order"],
                             current_predictor=c["predictor"], **DECK)


def loaded(c, seed):
    """A started simulation and its parameters."""
    Lx, Ly, x, y, u, q, m = plasma(c, seed)
    gamma = torch.sqrt(1 + (u * u).sum(1, keepdim=True)) if c["kind"] != "nonrel" and not c.get("two_stream") else 1.0
    v, P = (u / gamma).cpu().numpy(), (m[:, None] * u).cpu().numpy()
    if c["kind"] != "explicit":  # these methods centre the box on the origin and form P themselves
        x, y = x - 0.5 * Lx, y - 0.5 * Ly
    sim = up.Simulation(config(c, Lx, Ly))
    sim.set_particles(x.cpu().numpy(), y.cpu().numpy(), P, v, v, q.cpu().numpy(), m.cpu().numpy())
    sim.init_fields(False)
    return sim


def buffers(n):
    """Host buffers a driver keeps for the particle read-back (page-locked)."""
    pin = torch.cuda.is_available()
    return {k: torch.empty((n,) if k in "xy" else (n, 3), dtype=torch.float64, pin_memory=pin).numpy()
            for k in ("x", "y", "P", "v", "v_prev")}


def members(c):
    """The cases of an ensemble's runs."""
    n = c["runs"]
    for r in range(n):
        count = int(round(math.exp(math.log(c["least"]) + (math.log(c["most"]) - math.log(c["least"])) * r / (n - 1))))
        if c["method"] == "cn_orbit":
            m = implicit("", ENSEMBLE_NX_1D[r % 4], 1, count, 3, 0.1, c["steps"], two_stream=True)
            m["v0"] = 0.05 + 0.25 * ((7 * r) % n) / n
        else:
            m = explicit("", *ENSEMBLE_GRIDS[r % 4], count, steps=c["steps"])
        yield m


def prepare(case, seed):
    if case["kind"] == "ensemble":
        runs = list(members(case))
        sims = [loaded(m, 1000 * seed + r) for r, m in enumerate(runs)]
        total = sum(m["particles"] for m in runs)
        out, views, at = buffers(total), [], 0
        for m in runs:
            views.append({k: a[at:at + m["particles"]] for k, a in out.items()})
            at += m["particles"]
        return {"case": case, "ensemble": up.Ensemble(sims), "sims": sims, "views": views, "out": out}
    c = dict(case, v0=0.2) if case.get("two_stream") else case
    return {"case": case, "sim": loaded(c, seed), "out": buffers(c["particles"])}


def run(state):
    c = state["case"]
    if c["kind"] == "ensemble":
        state["ensemble"].step(c["steps"])
        for sim, view in zip(state["sims"], state["views"]):
            sim.get_particles(view)
        return {"particles": state["out"]}
    sim = state["sim"]
    if c["kind"] == "explicit":
        rows = {"diag": sim.step(c["steps"], c["stride"])}
    else:
        diag, info = sim.step_implicit(c["steps"])
        rows = {"diag": diag, "info": info}
    return {**rows, "fields": {k: sim.field(k) for k in FIELDS}, "particles": sim.get_particles(state["out"])}


def work(case):
    """Bytes: the particle state read and written once a step, the field state
    and the gathered fields once a step.  Flops: gather, push and deposit of
    each particle (for the implicit methods over the usual seven current
    iterations of three local ones) and the transforms."""
    if case["kind"] == "ensemble":
        all_ = [work(m) for m in members(case)]
        return {k: sum(w[k] for w in all_) for k in ("bytes", "flops")}
    n, N, K = case["particles"], case["nx"] * case["ny"], case["steps"]
    fft = 2.5 * N * max(1.0, math.log2(N))  # one real transform
    read_back = 88.0 * n + 64.0 * N
    if case["kind"] == "explicit":
        mixed = case["precision"] == "mixed"
        back = 2 if case["method"] == "bdf1" else 4
        return {"bytes": K * (n * (92.0 if mixed else 176.0) + N * (16.0 * 5 * (back + 1) + 88)) + read_back,
                "flops": K * (n * (9 * 11 * 2 + 9 * 3 * 2 + 110.0) + 14 * fft)}
    S = (case["order"] + 1) * (case["order"] + 1 if case["ny"] > 1 else 1)
    points = case["order"] + 1
    orbit = points * (S * 10 + 40.0) + S * 28.0       # one segment's shape sums and its node records
    deposit = points * (S * 2 + 20.0) + S * 6.0
    evals = 7
    local = 3 if case["kind"] == "implicit" else 1
    return {"bytes": K * (n * (112.0 + 112.0) + N * (16.0 * 18 + 64)) + read_back,
            "flops": K * evals * (n * (local * (orbit + 120.0) + deposit) + 8 * fft)}


# ---- the same results in plain torch, 64 bits ---------------------------------
def exact(case, seed):
    """What run() returns first, computed directly; None where it takes long."""
    if case["kind"] == "ensemble":
        runs = list(members(case))
        if case["method"] == "cn_orbit" and sum(m["particles"] for m in runs) * case["steps"] > 1.2e6:
            return None
        parts = [reference(m, 1000 * seed + r)["particles"] for r, m in enumerate(runs)]
        return {"particles": {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}}
    c = dict(case, v0=0.2) if case.get("two_stream") else case
    if c["particles"] * c["steps"] > (1.0e9 if c["kind"] == "explicit" else 2.5e6):
        return None
    return reference(c, seed)


class Grid:
    """Periodic grid: FFT wave numbers, derivatives, B-spline stencils."""

    def __init__(self, nx, ny, Lx, Ly, nyquist_k2=False, p2_modes=False):
        self.nx, self.ny, self.N, self.Lx, self.Ly = nx, ny, nx * ny, Lx, Ly
        self.hx, self.hy = Lx / nx, Ly / ny

        def modes(n, L, keep):
            k = torch.arange(n, dtype=torch.float64, device=device())
            k = torch.where(k < (n + 1) // 2, k, k - n)
            if n > 1 and not keep:
                k[n // 2] = 0.0
            if n == 1 and p2_modes:
                k[0] = -1.0
            return 2 * math.pi * k / L

        self.kx, self.ky = modes(nx, Lx, False)[:, None], modes(ny, Ly, False)[None, :]
        fx, fy = modes(nx, Lx, nyquist_k2)[:, None], modes(ny, Ly, nyquist_k2)[None, :]
        self.k2 = fx * fx + fy * fy
        keep = torch.ones(nx, ny, dtype=torch.float64, device=device())
        if nx > 1:
            keep[nx // 2, :] = 0
        if ny > 1:
            keep[:, ny // 2] = 0
        self.keep = keep

    def fft(self, f):
        return torch.fft.fft2(f.reshape(*f.shape[:-1], self.nx, self.ny) if f.shape[-1] == self.N else f)

    def real(self, s):
        return torch.fft.ifft2(s).real

    def nodes(self, sx, sy):
        """Node ids (n, S, S) of stencils whose first nodes are sx, sy."""
        def axis(s, n, size):
            return (s[:, None] + torch.arange(size, device=device())) % n
        return axis(sx[0], self.nx, sx[1])[:, :, None] * self.ny + axis(sy[0], self.ny, sy[1])[:, None, :]

    def add(self, out, ids, values):
        """out (N, k) += values (n, S, S, k) at ids (n, S, S)."""
        out.index_add_(0, ids.reshape(-1), values.reshape(-1, out.shape[1]))


def spline(order, f):
    """Weights and derivatives (n, order + 1) of the centred B-spline at
    stencil offset f, by the Cox-de Boor recurrence on integer knots."""
    t = f - 0.5 * (order - 1)  # position in the cell of the uniform knots, in [0, 1)
    w = [torch.ones_like(t)]
    low = None
    for p in range(1, order + 1):
        low = w
        new = []
        for a in range(p + 1):
            left = low[a - 1] * (t + p - a) / p if a > 0 else 0.0
            right = low[a] * (a + 1 - t) / p if a < p else 0.0
            new.append(left + right)
        w = new
    d = []
    for a in range(order + 1):
        d.append((low[a - 1] if a > 0 else 0.0) - (low[a] if a < order else 0.0) + torch.zeros_like(t))
    return torch.stack(w, 1), torch.stack(d, 1)


def chunks(n, size=1 << 20):
    for a in range(0, n, size):
        yield slice(a, min(a + size, n))


def to_host(d):
    return {k: (to_host(v) if isinstance(v, dict) else v.detach().cpu().numpy() if torch.is_tensor(v) else v)
            for k, v in d.items()}


def reference(c, seed):
    return to_host(reference_explicit(c, seed) if c["kind"] == "explicit" else reference_orbit(c, seed))


def reference_explicit(c, seed):
    Lx, Ly, x, y, u, q, m = plasma(c, seed)
    g = Grid(c["nx"], c["ny"], Lx, Ly, p2_modes=True)
    v = u / torch.sqrt(1 + (u * u).sum(1, keepdim=True))
    P, vp, dt, n = m[:, None] * u, v, 0.05, c["particles"]
    a = [1.0, -1.0] if c["method"] == "bdf1" else [1.5, -2.0, 0.5]
    b = [sum(a[i] * a[l - i] for i in range(len(a)) if 0 <= l - i < len(a)) for l in range(2 * len(a) - 1)]
    naive = c["charge"] == "naive"
    dA = g.hx * g.hy

    def stencil(s):
        xs, ys = x[s] / g.hx, y[s] / g.hy
        ix, iy = torch.floor(xs + 0.5), torch.floor(ys + 0.5)
        wx, wy = spline(2, xs - ix + 1.0)[0], spline(2, ys - iy + 1.0)[0]
        ids = g.nodes((ix.long() - 1, 3), (iy.long() - 1, 3))
        return ids, wx[:, :, None] * wy[:, None, :]

    def deposit():
        out = torch.zeros(g.N, 4, dtype=torch.float64, device=device())
        for s in chunks(n):
            ids, w = stencil(s)
            val = torch.cat([v[s], torch.ones_like(v[s][:, :1])], 1) * (q[s] / dA)[:, None]
            g.add(out, ids, w[..., None] * val[:, None, None, :])
        return out.T.reshape(4, g.nx, g.ny)

    dep = deposit()
    rho0 = g.fft(1.0 + dep[3])
    phi0 = torch.where(g.k2 > 0, rho0 / torch.where(g.k2 > 0, g.k2, torch.ones_like(g.k2)), torch.zeros_like(rho0))
    zero = torch.zeros_like(rho0)
    hist = [[f] * 5 for f in (phi0, zero, zero, zero, rho0)]  # newest first
    rows = np.full((c["steps"], 13), np.nan)
    scale = 1.0 / dt ** 2
    for step in range(1, c["steps"] + 1):
        x = torch.remainder(x + dt * v[:, 0], Lx)
        y = torch.remainder(y + dt * v[:, 1], Ly)
        x, y = torch.where(x >= Lx, x - Lx, x), torch.where(y >= Ly, y - Ly, y)
        dep = deposit()
        J = g.fft(dep[:3])
        divJ = 1j * (g.kx * J[0] + g.ky * J[1])
        if naive:
            rho = g.fft(1.0 + dep[3])
        else:
            rho = -(dt * divJ + sum(a[l] * hist[4][l - 1] for l in range(1, len(a)))) / a[0]
        den = scale * b[0] + g.k2
        new = []
        for f, src in enumerate((rho, J[0], J[1], J[2])):
            new.append((src - sum(scale * b[l] * hist[f][l - 1] for l in range(1, len(b)))) / den)
        phi, A = new[0], new[1:]
        hist = [[fn] + h[:-1] for fn, h in zip(new + [rho], hist)]
        spec = A + [1j * g.kx * phi, 1j * g.ky * phi]
        for comp in A:
            spec += [1j * g.kx * comp, 1j * g.ky * comp]
        F = g.real(torch.stack(spec)).reshape(11, g.N).T.contiguous()
        v_new, P_new = torch.empty_like(v), P.clone()
        for s in chunks(n):
            ids, w = stencil(s)
            G = (F[ids] * w[..., None]).sum((1, 2))
            vs = 2 * v[s] - vp[s]
            for d in range(2):
                force = (G[:, [5 + d, 7 + d, 9 + d]] * vs).sum(1) - G[:, 3 + d]
                P_new[s, d] += q[s] * dt * force
            p = P_new[s] - q[s][:, None] * G[:, :3]
            v_new[s] = p / torch.sqrt((p * p).sum(1) + m[s] ** 2)[:, None]
        v, vp, P = v_new, v, P_new
        if step % c["stride"] == 0 or step == c["steps"]:
            ddt = [sum(a[l] * h[l] for l in range(len(a))) / dt for h in hist]
            E = [-1j * g.kx * phi - ddt[1], -1j * g.ky * phi - ddt[2], -ddt[3]]
            B = [1j * g.ky * A[2], -1j * g.kx * A[2], 1j * (g.kx * A[1] - g.ky * A[0])]
            gauge = ddt[0] + 1j * (g.kx * A[0] + g.ky * A[1])
            gauss = 1j * (g.kx * E[0] + g.ky * E[1]) - rho
            f = g.real(torch.stack([gauge, gauss, ddt[4] + divJ, *E, *B, rho]))
            rms = lambda t: float(t.square().sum().div(g.N).sqrt())  # noqa: E731
            gam = 1 / torch.sqrt(torch.clamp(1 - (v * v).sum(1), min=1e-14))
            fe = 0.5 * float(f[3:9].square().sum()) * dA
            ke = float(((gam - 1) * m).sum())
            rows[step - 1] = [rms(f[0]), rms(f[1]), rms(f[2]), rms(f[8]), rms(f[6:9]), rms(f[3:6]), rms(f[9]),
                              rms(dep[:3]), fe, ke, fe + ke, float((v * v).sum(1).max().sqrt()), float(gam.mean())]
    fields = dict(zip(FIELDS, [g.real(h[0]) for h in hist] + [dep[0], dep[1], dep[2]]))
    return {"diag": rows, "fields": fields, "particles": {"x": x, "y": y, "P": P, "v": v, "v_prev": vp}}


def reference_orbit(c, seed):
    """The implicit methods: the orbit equations iterated to convergence."""
    rel = c["kind"] == "implicit"
    Lx, Ly, x, y, u, q, m = plasma(c, seed)
    x, y = x - 0.5 * Lx, y - 0.5 * Ly
    order, dt, n = c["order"], c["dt"], c["particles"]
    S = order + 1
    g = Grid(c["nx"], c["ny"], Lx, Ly, nyquist_k2=not rel)
    keep = g.keep if rel else torch.ones_like(g.keep)
    off = 0.5 * (order - 1)
    gl = [torch.tensor(t, device=device()) for t in np.polynomial.legendre.leggauss(S)]
    gs, gw = 0.5 * (gl[0] + 1), 0.5 * gl[1]
    dV = g.hx * g.hy
    v = u
    if rel:
        if not c.get("two_stream"):
            v = u / torch.sqrt(1 + (u * u).sum(1, keepdim=True))
        P = (m / torch.sqrt(1 - (v * v).sum(1)))[:, None] * v
    else:
        P = m[:, None] * v

    def axis(pos, L, h, il=None):
        t = (pos + 0.5 * L) / h
        i = torch.floor(t - off) if il is None else il
        w, d = spline(order, t - i)
        return i.long(), w, d / h

    def at(s, px, py, fields):
        ix, wx, _ = axis(px, Lx, g.hx)
        iy, wy, _ = axis(py, Ly, g.hy)
        ids = g.nodes((ix, S), (iy, S))
        return (fields[ids] * (wx[:, :, None] * wy[:, None, :])[..., None]).sum((1, 2))

    def knots(p0, d, L, h):
        """Orbit fractions (n, K) where the orbit crosses a knot of one axis."""
        u0, du = (p0 + 0.5 * L) / h - off, d / h
        lo = torch.minimum(u0, u0 + du)
        K = int(torch.ceil(du.abs().max()).item()) + 1
        s = (torch.floor(lo)[:, None] + 1 + torch.arange(K, device=device()) - u0[:, None]) / du[:, None]
        return torch.where((s > 0) & (s < 1), s, torch.ones_like(s))

    def segments(s, d):
        b = torch.cat([torch.zeros_like(x[s])[:, None], knots(x[s], d[:, 0], Lx, g.hx), knots(y[s], d[:, 1], Ly, g.hy),
                       torch.ones_like(x[s])[:, None]], 1).sort(1)[0]
        for k in range(b.shape[1] - 1):
            on = (b[:, k + 1] > b[:, k]).nonzero().squeeze(1)
            if on.numel():
                a, ln = b[on, k], b[on, k + 1] - b[on, k]
                mid = a + 0.5 * ln
                ix = torch.floor((x[s][on] + mid * d[on, 0] + 0.5 * Lx) / g.hx - off)
                iy = torch.floor((y[s][on] + mid * d[on, 1] + 0.5 * Ly) / g.hy - off)
                ids = g.nodes((ix.long(), S), (iy.long(), S))
                pts = []
                for k2 in range(S):
                    t = a + ln * gs[k2]
                    _, wx, dx = axis(x[s][on] + t * d[on, 0], Lx, g.hx, ix)
                    _, wy, dy = axis(y[s][on] + t * d[on, 1], Ly, g.hy, iy)
                    pts.append((t, ln * gw[k2], wx, dx, wy, dy))
                yield on, ids, pts

    def orbit_current(vb):
        out = torch.zeros(g.N, 3, dtype=torch.float64, device=device())
        for s in chunks(n, 1 << 18):
            for on, ids, pts in segments(s, dt * vb[s]):
                w = sum(wq[:, None, None] * wx[:, :, None] * wy[:, None, :] for _, wq, wx, _, wy, _ in pts)
                g.add(out, ids, w[..., None] * (vb[s][on] * (q[s][on] / dV)[:, None])[:, None, None, :])
        return out.T.reshape(3, g.nx, g.ny)

    def averages(s, vb, F):
        """Orbit averages of grad phi (n, 2) and of dA_c/dx_d (n, 3, 2)."""
        k = s.stop - s.start
        gp = torch.zeros(k, 2, dtype=torch.float64, device=device())
        D = torch.zeros(k, 3, 2, dtype=torch.float64, device=device())
        for on, ids, pts in segments(s, dt * vb):
            f = F[ids]
            for t, wq, wx, dx, wy, dy in pts:
                sh = wx[:, :, None] * wy[:, None, :]
                gp.index_add_(0, on, wq[:, None] * (f[..., :2] * sh[..., None]).sum((1, 2)))
                A = (1 - t)[:, None, None, None] * f[..., 2:5] + t[:, None, None, None] * f[..., 5:8]
                Dx = (A * (dx[:, :, None] * wy[:, None, :])[..., None]).sum((1, 2))
                Dy = (A * (wx[:, :, None] * dy[:, None, :])[..., None]).sum((1, 2))
                D.index_add_(0, on, wq[:, None, None] * torch.stack([Dx, Dy], 2))
        return gp, D

    def gam(p, ms):
        return torch.sqrt(1 + (p * p).sum(1) / ms ** 2)[:, None]

    def push(s, vb, F):
        """One map evaluation: end position, momentum, velocity, mapped vbar."""
        x1 = torch.remainder(x[s] + dt * vb[:, 0] + 0.5 * Lx, Lx) - 0.5 * Lx
        y1 = torch.remainder(y[s] + dt * vb[:, 1] + 0.5 * Ly, Ly) - 0.5 * Ly
        A1 = at(s, x1, y1, F[:, 5:8])
        gp, D = averages(s, vb, F)
        gp3 = torch.cat([gp, torch.zeros_like(gp[:, :1])], 1)
        qs, ms = q[s][:, None], m[s]
        if not rel:
            DTv = torch.einsum("ncd,nc->nd", D, vb)
            P1 = P[s] + dt * qs * (torch.cat([DTv, torch.zeros_like(gp[:, :1])], 1) - gp3)
            v1 = (P1 - qs * A1) / ms[:, None]
            return x1, y1, P1, v1, 0.5 * (v1 + v[s])
        A0 = at(s, x[s], y[s], F[:, 2:5])
        Am = 0.5 * (A0 + A1)
        Dv = torch.einsum("ncd,nd->nc", D, vb[:, :2])
        Bf = torch.stack([D[:, 2, 1], -D[:, 2, 0], D[:, 1, 0] - D[:, 0, 1]], 1)
        kick = 0.5 * qs * dt * (Dv - gp3)
        pm = P[s] - qs * Am + kick
        um, tau = pm / ms[:, None], qs * dt / (2 * ms[:, None]) * Bf
        g2 = 1 + (um * um).sum(1)
        sig, ut, t2 = g2 - (tau * tau).sum(1), (um * tau).sum(1), (tau * tau).sum(1)
        gh = torch.sqrt(torch.clamp(0.5 * (sig + torch.sqrt(sig ** 2 + 4 * (t2 + ut ** 2))), min=1.0))
        tv = tau / gh[:, None]
        up_ = um + torch.linalg.cross(um, tv)
        upl = um + torch.linalg.cross(up_, 2 / (1 + (tv * tv).sum(1, keepdim=True)) * tv)
        pp = upl * ms[:, None]
        P1 = pp + qs * Am + kick
        pe, p0 = P1 - qs * A1, P[s] - qs * A0
        v1 = pe / (ms[:, None] * gam(pe, ms))
        vm = 0.5 * ((pm + p0) / (ms[:, None] * (gam(pm, ms) + gam(p0, ms))) +
                    (pe + pp) / (ms[:, None] * (gam(pe, ms) + gam(pp, ms))))
        return x1, y1, P1, v1, vm

    # start: charge and current of the loaded particles, phi from Poisson
    out = torch.zeros(g.N, 4, dtype=torch.float64, device=device())
    for s in chunks(n):
        ix, wx, _ = axis(x[s], Lx, g.hx)
        iy, wy, _ = axis(y[s], Ly, g.hy)
        val = torch.cat([v[s], torch.ones_like(v[s][:, :1])], 1) * (q[s] / dV)[:, None]
        g.add(out, g.nodes((ix, S), (iy, S)), (wx[:, :, None] * wy[:, None, :])[..., None] * val[:, None, None, :])
    dep = out.T.reshape(4, g.nx, g.ny)
    J = g.real(g.fft(dep[:3]) * keep)
    rho = g.fft(dep[3]) * keep
    rho[0, 0] = 0
    inv = torch.where(g.k2 > 0, 1 / torch.where(g.k2 > 0, g.k2, torch.ones_like(g.k2)), torch.zeros_like(g.k2))
    phi, psi = rho * inv * keep, torch.zeros_like(rho)
    A = [torch.zeros_like(rho) for _ in range(3)]
    U = [torch.zeros_like(rho) for _ in range(3)]
    theta = 0.25 * dt * dt * g.k2

    def cn(f, fd, src):
        return (keep * ((1 - theta) * f + dt * fd + 0.5 * dt * dt * src) / (1 + theta),
                keep * ((1 - theta) * fd - dt * g.k2 * f + dt * src) / (1 + theta))

    rows = np.empty((c["steps"], len(up.IMPLICIT_DIAG_COLUMNS)))
    for step in range(c["steps"]):
        vb = v.clone()
        for it in range(16):
            Jh = g.fft(J if it else (J if rel else orbit_current(vb))) * keep
            rho1 = keep * (rho - dt * 1j * (g.kx * Jh[0] + g.ky * Jh[1]))
            rho1[0, 0] = 0
            phi1, psi1 = cn(phi, psi, 0.5 * (rho + rho1))
            phi1[0, 0] = psi1[0, 0] = 0
            AU = [cn(A[k], U[k], Jh[k]) for k in range(3)]
            F = g.real(torch.stack([0.5j * g.kx * (phi + phi1), 0.5j * g.ky * (phi + phi1), *A,
                                    *[a[0] for a in AU]])).reshape(8, g.N).T.contiguous()
            x1, y1, P1, v1, vb1 = (torch.empty_like(t) for t in (x, y, P, v, v))
            for s in chunks(n, 1 << 18):
                w = vb[s]
                for _ in range(12 if rel else 1):
                    r = push(s, w, F)
                    moved, w = float((r[4] - w).abs().max()), r[4]
                    if moved < 1e-16:
                        break
                x1[s], y1[s], P1[s], v1[s], vb1[s] = r
            change = float((vb1 - vb).square().mean().sqrt())
            vb = vb1
            Jn = orbit_current(vb)
            if rel:
                Jn = g.real(g.fft(Jn) * keep)
            done = float((Jn - J).abs().max()) < 2e-15 * float(Jn.abs().max()) + 1e-300
            J = Jn
            if it and (done or change < 1e-17):
                break
        x, y, P, vp, v = x1, y1, P1, v, v1
        phi, psi, rho, A, U = phi1, psi1, rho1, [a[0] for a in AU], [a[1] for a in AU]
        E = [-1j * g.kx * phi - U[0], -1j * g.ky * phi - U[1], -U[2]]
        B = [1j * g.ky * A[2], -1j * g.kx * A[2], 1j * (g.kx * A[1] - g.ky * A[0])]
        divE, divA = 1j * (g.kx * E[0] + g.ky * E[1]), 1j * (g.kx * A[0] + g.ky * A[1])
        f = g.real(torch.stack([*E, *B, divE, divA, psi, rho]))
        rms = lambda t: float(t.square().mean().sqrt())  # noqa: E731
        gs_, ga = f[6] - f[9], f[8] + f[7]
        beta2 = (v * v).sum(1)
        ke = float((m * (1 / torch.sqrt(1 - beta2) - 1)).sum()) if rel else float((0.5 * m * beta2).sum())
        fe = 0.5 * float(f[:6].square().sum()) * dV
        mx, my = (1 % g.nx, 0), (0, 1 % g.ny)
        em, bm = complex(E[0][mx]) / g.N, complex(B[2][my]) / g.N
        d = {"gauss_rms": rms(gs_), "gauss_max": float(gs_.abs().max()), "divE_rms": rms(f[6]),
             "sigma1_rho_rms": rms(f[9]), "gauge_rms": rms(ga), "gauge_max": float(ga.abs().max()),
             "psi_over_kappa2_rms": rms(f[8]), "divA_rms": rms(f[7]), "field_energy": fe, "kinetic_energy": ke,
             "total_energy": fe + ke, "rho_mode": abs(complex(rho[mx])) / g.N, "E_mode_re": em.real,
             "E_mode_im": em.imag, "E_mode_abs": abs(em), "Bz_y_mode_re": bm.real, "Bz_y_mode_im": bm.imag,
             "Bz_y_mode_abs": abs(bm), "mean_rho": float(f[9].mean())}
        d["gauss_normalization_rms"] = d["divE_rms"] + d["sigma1_rho_rms"]
        d["gauss_relative"] = d["gauss_rms"] / max(d["gauss_normalization_rms"], 1e-300)
        d["gauge_normalization_rms"] = d["psi_over_kappa2_rms"] + d["divA_rms"]
        d["gauge_relative"] = d["gauge_rms"] / max(d["gauge_normalization_rms"], 1e-300)
        rows[step] = [d[k] for k in up.IMPLICIT_DIAG_COLUMNS]
    fields = dict(zip(FIELDS, [g.real(t) for t in (phi, *A, rho)] + [J[0], J[1], J[2]]))
    return {"diag": rows, "info": None, "fields": fields,
            "particles": {"x": x, "y": y, "P": P, "v": v, "v_prev": vp}}
