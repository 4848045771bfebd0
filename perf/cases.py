"""The work that a user has this framework do, as cases to be timed.

Every case is one call (or the short sequence of calls) of a user's program on a solver it has built:

* ``steps``      leap-frog steps of a prepared solver: ``run`` (from an initial H), or ``run_with_io`` with the
                 beam current and the Ez window of every step going through pinned host memory;
* ``wakesolve``  the whole wake computation of a cavity: steps with the beam, then wake potential and impedance;
* ``emsolve``    a plane wave through a periodic cell into a PML;
* ``post``       ``WakeSolver.solve`` on an Ez history that is already there (another frequency range, other
                 skipped cells, a history of an earlier run);
* ``adjoint``    one iteration of an optimiser: new material parameters, loss, gradient;
* ``batch``      many cavities of a parameter scan stepped together.

Grids are boxes of 1 mm cells with a cavity and a beam pipe in a PEC or conductive wall.  Sizes run from the
tests' smallest grid (16x16x24) to the benchmark's (256x256x512), and are as often odd as even: a grid's cell
counts follow from a geometry and a cell size, not from what a kernel likes.

``exact`` restates the same equations with torch in 64 bits on whole arrays.
"""

import functools

import numpy as np
import torch

C = 299792458.0
EPS0 = 8.8541878188e-12
MU0 = 1.25663706127e-06
CELL = 1e-3
DTYPES = {"f64": np.float64, "f32": np.float32, "f32c": np.float64}
STATE_BYTES = {"f64": 8, "f32": 4, "f32c": 6}   # f32c: float values and 16-bit compensation words

# faces (low x, y, z), (high x, y, z) and background of the wall
SETUPS = {
    # closed cavity in a perfect conductor
    "closed": (("pec", "pec", "pec"), ("pec", "pec", "pec"), "pec"),
    # beam pipe open at both ends
    "open": (("pec", "pec", "abc"), ("pec", "pec", "abc"), "pec"),
    # conductive wall, absorbing layers at both ends of the pipe
    "lossy": (("pec", "pec", "pml"), ("pec", "pec", "pml"), [1.0, 1.0, 1e4]),
    # the same with a poor conductor (the time step stays the grid's own)
    "absorber": (("pec", "pec", "pml"), ("pec", "pec", "pml"), [1.0, 1.0, 5.0]),
    # periodic cell, vacuum, open on one side of z
    "periodic": (("periodic", "periodic", "pec"), ("periodic", "periodic", "pml"), [1.0, 1.0]),
}
N_PML = 10


def listed():
    return [
        # the smallest whole run: a test cavity, a few hundred steps (launches and host work)
        dict(name="wakesolve_16x16x24_f64", kind="wakesolve", nx=16, ny=16, nz=24, dtype="f64", setup="closed",
             wakelength=0.06, sigmaz=0.004),
        # the 50x50x150 float32 cavity of the regression test, 1 m of wake
        dict(name="wakesolve_50x50x150_f32", kind="wakesolve", nx=50, ny=50, nz=150, dtype="f32", setup="closed",
             wakelength=0.6, sigmaz=0.0185),
        # the 40x40x80 cavity workload with open pipe ends
        dict(name="wakesolve_40x40x80_f64", kind="wakesolve", nx=40, ny=40, nz=80, dtype="f64", setup="open",
             wakelength=0.4, sigmaz=0.010),
        # the benchmark's grid, every step with its host traffic
        dict(name="steps_256x256x512_f64_io", kind="steps", nx=256, ny=256, nz=512, dtype="f64", setup="lossy",
             steps=8, io=True),
        # large runs in single precision and with the compensated state
        dict(name="steps_256x256x512_f32", kind="steps", nx=256, ny=256, nz=512, dtype="f32", setup="lossy",
             steps=8, io=False),
        dict(name="steps_224x224x448_f32c", kind="steps", nx=224, ny=224, nz=448, dtype="f32c", setup="open",
             steps=8, io=False),
        # ordinary grids whose sizes are what the geometry gave
        dict(name="steps_149x131x301_f64", kind="steps", nx=149, ny=131, nz=301, dtype="f64", setup="open",
             steps=16, io=False),
        dict(name="steps_101x99x203_f32", kind="steps", nx=101, ny=99, nz=203, dtype="f32", setup="lossy",
             steps=32, io=False),
        # a unit cell of a periodic structure
        dict(name="emsolve_96x96x240_f64", kind="emsolve", nx=96, ny=96, nz=240, dtype="f64", setup="periodic",
             steps=60),
        # wake potential and impedance of a long history
        dict(name="post_400x12000", kind="post", nz=400, nt=12000, skip=0, dtype="f64"),
        # gradient of an impedance band with respect to the materials of a block
        dict(name="adjoint_40x40x80_f64", kind="adjoint", nx=40, ny=40, nz=80, dtype="f64", setup="closed",
             block=16, steps=600),
        # a scan of cavities, compensated state
        dict(name="batch_8_f32c", kind="batch", count=8, dtype="f32c", steps=900, nx=40, nz=96, spread=24),
    ]


def _log(rng, a, b):
    return int(round(a * (b / a) ** rng.random()))


def draw(rng):
    kind = rng.choice(["steps"] * 8 + ["wakesolve"] * 5 + ["emsolve"] * 2 + ["post"] * 2 + ["adjoint", "batch"])
    if kind == "steps":
        dtype = rng.choice(["f64", "f64", "f32", "f32c"])
        nx, ny, nz = _log(rng, 24, 256), _log(rng, 24, 256), _log(rng, 48, 512)
        # a multiple of 8 as often as what the geometry gave: users choose such sizes too
        if rng.random() < 0.4:
            nx, ny = max(24, nx // 8 * 8), max(24, ny // 8 * 8)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, setup=rng.choice(["lossy", "open", "closed"]),
                    steps=rng.choice([4, 6, 8]) if nx * ny * nz > 4_000_000 else rng.choice([8, 16, 32]),
                    io=rng.random() < 0.25)
    if kind == "wakesolve":
        nx, ny, nz = _log(rng, 14, 64), _log(rng, 14, 64), _log(rng, 24, 160)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=rng.choice(["f64", "f64", "f32", "f32c"]),
                    setup=rng.choice(["closed", "open", "absorber"]), wakelength=round(0.05 + 0.35 * rng.random(), 3),
                    sigmaz=round(0.004 + 0.008 * rng.random(), 4))
    if kind == "emsolve":
        nx = _log(rng, 16, 110)
        return dict(kind=kind, nx=nx, ny=_log(rng, 16, 110), nz=_log(rng, 48, 260),
                    dtype=rng.choice(["f64", "f64", "f32"]), setup="periodic", steps=rng.randrange(40, 80))
    if kind == "post":
        return dict(kind=kind, nz=_log(rng, 60, 420), nt=_log(rng, 2000, 12000), skip=rng.choice([0, 0, 7]),
                    dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "adjoint":
        return dict(kind=kind, nx=_log(rng, 28, 44), ny=_log(rng, 28, 44), nz=_log(rng, 48, 80), dtype="f64",
                    setup="closed", block=rng.choice([8, 11, 16]), steps=rng.randrange(520, 620))
    return dict(kind=kind, count=rng.randrange(4, 9), dtype="f32c", steps=rng.randrange(800, 950),
                nx=_log(rng, 28, 44) // 4 * 4, nz=_log(rng, 64, 100), spread=rng.choice([8, 16, 24]))


# ------------------------------------------------------------------ geometry
def _bounds(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (-nx * CELL / 2, nx * CELL / 2, -ny * CELL / 2, ny * CELL / 2, -nz * CELL / 2, nz * CELL / 2)


def _edges(case):
    b = _bounds(case)
    return tuple(np.linspace(b[2 * a], b[2 * a + 1], case[n] + 1) for a, n in enumerate(("nx", "ny", "nz")))


def _any_corner(m):
    for a in range(3):
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        m = m[tuple(lo)] | m[tuple(hi)]
    return m


@functools.lru_cache(maxsize=4)
def _cavity(nx, ny, nz):
    """Vacuum cells: a box cavity of 0.6 of the transverse size and 0.3 of the length, a square pipe along z."""
    x, y, z = _edges(dict(nx=nx, ny=ny, nz=nz))
    box = ((np.abs(x) <= 0.3 * nx * CELL)[:, None, None] & (np.abs(y) <= 0.3 * ny * CELL)[None, :, None]
           & (np.abs(z) <= 0.15 * nz * CELL)[None, None, :])
    pipe = (np.abs(x) <= 0.12 * nx * CELL + 2 * CELL)[:, None] & (np.abs(y) <= 0.12 * ny * CELL + 2 * CELL)[None, :]
    return _any_corner(box | pipe[:, :, None])


def _beam_args(case, seed):
    r = np.random.default_rng(seed)
    return dict(q=float(1e-9 * (0.5 + r.random())), sigmaz=case.get("sigmaz", 0.01), beta=case.get("beta", 1.0),
                xsource=float(CELL * (r.random() - 0.5)), ysource=float(CELL * (r.random() - 0.5)),
                xtest=float(CELL * (r.random() - 0.5)), ytest=float(CELL * (r.random() - 0.5)))


def _solver(case, seed):
    import wakis_b200 as wb
    low, high, bg = SETUPS[case["setup"]]
    g = wb.GridFIT3D(*_bounds(case), case["nx"], case["ny"], case["nz"], verbose=0)
    if case["setup"] != "periodic":
        g.add_solid("cavity", _cavity(case["nx"], case["ny"], case["nz"]), "vacuum")
    if case.get("liner"):
        g.add_solid("liner", _liner(case), [10.0, 1.0, 1.0])
    w = wb.WakeSolver(save=False, verbose=0, **_beam_args(case, seed))
    return wb.SolverFIT3D(g, w, bc_low=list(low), bc_high=list(high), use_stl=case["setup"] != "periodic", bg=bg,
                          n_pml=N_PML, dtype=DTYPES[case["dtype"]], verbose=0,
                          precision="fp32c" if case["dtype"] == "f32c" else None)


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _initial_h(case, seed):
    n3 = 3 * case["nx"] * case["ny"] * case["nz"]
    return torch.randn(n3, generator=_generator(seed), device=_device(), dtype=torch.float32)


def _io_lines(case, seed):
    r = np.random.default_rng(seed + 1)
    k = np.arange(case["nz"])[None, :] - 0.4 * case["nz"] - np.arange(case["steps"])[:, None]
    return (1e6 * (0.5 + r.random()) * np.exp(-k ** 2 / 200.0) * (1 + 0.1 * r.standard_normal(k.shape)))


# design block of the adjoint cases: in the middle of the cavity, beside the beam
def _block(case):
    m = np.zeros((case["nx"], case["ny"], case["nz"]), bool)
    b = case["block"]
    i0, j0, k0 = case["nx"] // 2 - b // 2, case["ny"] // 2 - b // 2, case["nz"] // 2 - b // 2
    m[i0:i0 + b, j0:j0 + b, k0:k0 + b] = True
    return m


def _params(case, seed):
    r = np.random.default_rng(seed + 2)
    n = case["block"] ** 3
    return r.uniform(1.0, 10.0, n), r.uniform(0.0, 10.0, n)


F_BAND = (0.5e9, 3e9)


# the instances of a batch: cavities of several sizes with a lossy liner
def _instances(case, seed):
    r = np.random.default_rng(case["count"] * 1000 + case["nx"])
    s = np.random.default_rng(seed)
    out = []
    for q in range(case["count"]):
        n = case["nx"] + 4 * int(r.integers(0, case["spread"] // 4 + 1))
        out.append(dict(nx=n, ny=n, nz=case["nz"] + int(r.integers(0, case["spread"])), dtype=case["dtype"],
                        setup="open", sigmaz=0.006, beta=float(0.8 + 0.2 * r.random()), liner=True,
                        seed=int(s.integers(1 << 30))))
    return out


def _liner(case):
    """Cells of the outer cavity region near one end (absorber ring)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = np.zeros((nx, ny, nz), bool)
    a, b = int(0.25 * nx), int(0.12 * nz)
    m[a:nx - a, a:ny - a, nz // 2 + b // 2:nz // 2 + b] = True
    c = int(0.35 * nx)
    m[c:nx - c, c:ny - c] = False
    return m


def _wakelength(n_steps, dt, w, length):
    """The wake length whose run has n_steps steps."""
    return (n_steps + 0.5) * dt * w.v - w.ti * w.v - length


# ----------------------------------------------------------------- interface
def prepare(case, seed):
    kind = case["kind"]
    if kind == "post":
        return _prepare_post(case, seed)
    if kind == "batch":
        return {"case": case, "solvers": [_solver(c, c["seed"]) for c in _instances(case, seed)]}
    s = _solver(case, seed)
    state = {"case": case, "solver": s}
    if kind == "steps":
        if case["io"]:
            pin = torch.cuda.is_available()
            lines = torch.as_tensor(_io_lines(case, seed))
            cap = torch.float32 if case["dtype"] == "f32" else torch.float64
            state["lines"] = lines.to(cap).pin_memory() if pin else lines.to(cap)
            out = torch.zeros((case["steps"], 9, case["nz"]), dtype=cap)
            state["out"] = out.pin_memory() if pin else out
        else:
            s.H.fromarray(_initial_h(case, seed))
    elif kind == "emsolve":
        import wakis_b200 as wb
        amp, f = _wave(case, seed)
        state["source"] = wb.sources.PlaneWave(zs=0, f=f, amplitude=amp, nodes=3)
    elif kind == "adjoint":
        from wakis_b200.adjoint import ImpedanceDesign
        state["design"] = ImpedanceDesign(s, _block(case), f_band=F_BAND, n_steps=case["steps"])
        state["params"] = _params(case, seed)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "post":
        w = state["wake"]
        w.solve(compute_plane="both")
        return _wake_results(w)
    if kind == "batch":
        from wakis_b200.batch import BatchedWakeSolve
        for s in state["solvers"]:
            s.reset_fields()
        BatchedWakeSolve(state["solvers"], case["steps"], tune=False).run()
        return [_wake_results(s.wake) for s in state["solvers"]]
    s = state["solver"]
    if kind == "steps":
        if case["io"]:
            s.run_with_io(state["lines"], state["out"])
            return {"E": s.E.toarray(), "H": s.H.toarray(), "ez": state["out"]}
        s.run(case["steps"])
        return {"E": s.E.toarray(), "H": s.H.toarray()}
    s.reset_fields()
    if kind == "wakesolve":
        s.wakesolve(wakelength=case["wakelength"])
        return dict(_wake_results(s.wake), E=s.E.toarray(), H=s.H.toarray())
    if kind == "emsolve":
        s.emsolve(case["steps"], source=state["source"])
        return {"E": s.E.toarray(), "H": s.H.toarray()}
    d = state["design"]
    d.set_params(*state["params"])
    loss = d.forward()
    g_eps, g_sigma = d.backward()
    return {"loss": loss, "eps": g_eps, "sigma": g_sigma}


def work(case):
    """Bytes and operations that the pass cannot do without: per cell and step the six components of E and H read
    and written once; the history read once and the sums over it."""
    kind = case["kind"]
    if kind == "post":
        ns = case["nt"]
        size = 4 if case["dtype"] == "f32" else 8
        return {"bytes": 9 * case["nz"] * ns * size, "flops": 18 * case["nz"] * ns}
    if kind == "batch":
        cells = sum(c["nx"] * c["ny"] * c["nz"] for c in _instances(case, 0))
        return {"bytes": 12 * STATE_BYTES[case["dtype"]] * cells * case["steps"], "flops": 60 * cells * case["steps"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "wakesolve":
        steps = _wake_steps(case)
    elif kind == "adjoint":
        steps = 3 * case["steps"]          # forward, forward again from checkpoints, reverse
    else:
        steps = case["steps"]
    return {"bytes": 12 * STATE_BYTES[case["dtype"]] * cells * steps, "flops": 60 * cells * steps}


def _wake_results(w):
    return {k: getattr(w, k) for k in ("WP", "WPx", "WPy", "Z", "Zx", "Zy")}


def _wave(case, seed):
    r = np.random.default_rng(seed)
    return float(100.0 * (0.5 + r.random())), float(C / (0.25 * case["nz"] * CELL) * (0.8 + 0.4 * r.random()))


# ------------------------------------------- a history without its time steps
def _post_axes(case):
    nz, dt = case["nz"], 0.5 * CELL / (C * np.sqrt(3.0))
    sigmaz = 0.004
    ti = 8.548921333333334 * sigmaz / C
    z = (np.arange(nz) + 0.5) * CELL - 0.5 * nz * CELL
    wakelength = float(case["nt"] * dt * C - (z.max() - z.min()) - ti * C)
    x = (np.arange(3) - 1.0) * CELL
    return z, x, dt, sigmaz, ti, wakelength


def _post_history(case, seed):
    """Decaying random Ez on the 3x3 window."""
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    h = torch.randn((9, case["nz"], case["nt"]), generator=_generator(seed), device=_device(), dtype=dt)
    return h.mul_(torch.exp(-3.0 * torch.arange(case["nt"], device=_device()) / case["nt"]).to(dt))


def _prepare_post(case, seed):
    import wakis_b200 as wb
    z, x, dt, sigmaz, ti, wakelength = _post_axes(case)
    w = wb.WakeSolver(wakelength=wakelength, sigmaz=sigmaz, skip_cells=case["skip"], save=False, verbose=0,
                      **{k: v for k, v in _beam_args(case, seed).items() if k != "sigmaz"})
    w.xf, w.yf, w.zf = x, x, z
    w.dz = np.full(case["nz"], CELL)
    w.t = np.arange(0, case["nt"] * dt, dt)
    w.set_history(_post_history(case, seed), n_steps=case["nt"])
    return {"case": case, "wake": w}


# ------------------------------------------------------- 64-bit restatement
def exact(case, seed):
    kind = case["kind"]
    if kind == "post":
        z, x, dt, sigmaz, ti, wl = _post_axes(case)
        return _wake_exact(_post_history(case, seed).double(), np.arange(0, case["nt"] * dt, dt), z,
                           np.full(case["nz"], CELL), x, x, wl, sigmaz, ti, _beam_args(case, seed)["q"],
                           case["skip"])
    if kind == "batch":
        return [_wakesolve_exact(c, c["seed"], steps=case["steps"])[0] for c in _instances(case, seed)]
    if kind == "wakesolve":
        res, f = _wakesolve_exact(case, seed)
        return dict(res, E=f.flat(f.E), H=f.flat(f.H))
    if kind == "adjoint":
        return _adjoint_exact(case, seed)
    f = _Fit(case)
    if kind == "steps":
        if case["io"]:
            lines = torch.as_tensor(_io_lines(case, seed), device=f.dev)
            if case["dtype"] == "f32":
                lines = lines.float().double()
            i, j = f.cell(0.0, 0.0)
            ez = torch.zeros((case["steps"], 9, case["nz"]), dtype=torch.float64, device=f.dev)
            for n in range(case["steps"]):
                ez[n] = f.window(i, j)
                f.step(line=(i, j, lines[n]))
            return {"E": f.flat(f.E), "H": f.flat(f.H), "ez": ez}
        h = _initial_h(case, seed).double().view(3, f.N)
        f.H = [h[d].clone() for d in range(3)]
        f.ghosts()
        for n in range(case["steps"]):
            f.step()
        return {"E": f.flat(f.E), "H": f.flat(f.H)}
    amp, freq = _wave(case, seed)
    w = 2 * np.pi * freq
    plane = case["nx"] * case["ny"]
    for n in range(case["steps"]):
        t = n * f.dt
        wave = np.cos(w * t) if t <= 3 / freq else 0.0
        f.H[1][:plane] = -amp * wave
        f.E[0][:plane] = amp * wave / (w / C / (MU0 * C))
        if n == 0:
            f.ghosts()
        f.step()
    return {"E": f.flat(f.E), "H": f.flat(f.H)}


def _wake_dt(case):
    dt = 0.5 / (C * np.sqrt(3.0 / CELL ** 2))
    return float(np.float32(dt)) if case["dtype"] == "f32" else dt


def _wake_steps(case):
    """About the steps of the run (the exact count follows from the solver's own time step)."""
    length = (case["nz"] - 1) * CELL
    return int((case["wakelength"] + 8.548921333333334 * case["sigmaz"] + length) / C / _wake_dt(case))


class _Fit:
    """The finite-integration update on whole arrays in 64 bits: separable metrics, the flat-offset difference
    operators of the method (a step past the end of a row lands on the next row), face masks in the order x, y, z
    (a later face replaces an earlier one), absorbing layers as graded conductivity."""

    def __init__(self, case, eps=None, sigma=None, block=None):
        self.dev = _device()
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.shape, self.N = (nz, ny, nx), nx * ny * nz
        low, high, bg = SETUPS[case["setup"]]
        ex, ey, ez = edges = _edges(case)
        self.x, self.y, self.z = (a[:-1] + np.diff(a) / 2 for a in edges)
        L = [np.diff(a) for a in edges]
        tL = []
        for a in edges:
            m = np.append((a[1:] + a[:-1]) / 2, 0.0)
            m[-1] = m[-2]
            tL.append(m[1:] - m[:-1])
        inv = lambda a, b: np.divide(1.0, np.multiply.outer(a, b), out=np.zeros((len(a), len(b))),  # noqa: E731
                                     where=np.multiply.outer(a, b) != 0)
        pair = ((1, 2), (0, 2), (0, 1))
        iA = [inv(L[a], L[b]) for a, b in pair]
        itA = [inv(tL[a], tL[b]) for a, b in pair]
        for a in range(3):
            if (low[a] == "periodic" and high[a] == "periodic") or high[a] == "abc":
                tL[a][-1] = L[a][0]
                for d in range(3):
                    if d != a:
                        ix = [slice(None)] * 2
                        ix[pair[d].index(a)] = -1
                        jx = list(ix)
                        jx[pair[d].index(a)] = 0
                        itA[d][tuple(ix)] = iA[d][tuple(jx)]
        self.dz, self.L = L[2], L
        # materials: background, vacuum cavity, liner, absorbing layers
        eb, mb = (np.inf, 1.0) if bg == "pec" else bg[:2]
        sb = bg[2] if bg != "pec" and len(bg) == 3 else 0.0
        self.conductive = sb > 0 or "pml" in low + high or bool(case.get("liner"))
        ieps = np.full((nx, ny, nz), 1.0 / (eb * EPS0))
        sig = np.full((nx, ny, nz), sb)
        if case["setup"] != "periodic":
            m = _cavity(nx, ny, nz)
            ieps[m], sig[m] = 1.0 / EPS0, 0.0
        if case.get("liner"):
            m = _liner(case)
            ieps[m], sig[m] = 1.0 / (10.0 * EPS0), 1.0
        for side, b in (("lo", low[2]), ("hi", high[2])):
            if b != "pml":
                continue
            grade = np.geomspace(10.0, 5e-3, N_PML)
            probe = (nx // 2, ny // 2, N_PML + 1 if side == "lo" else nz - (N_PML + 1))
            e0, s0 = ieps[probe], sig[probe]
            for p in range(N_PML):
                k = p if side == "lo" else nz - 1 - p
                ieps[:, :, k], sig[:, :, k] = e0, s0 + (s0 if s0 >= 1 else 1.0) * grade[p]
        dt = 0.5 / (C * np.sqrt(sum(1 / np.min(a) ** 2 for a in L)))
        real = np.float32 if case["dtype"] == "f32" else np.float64
        self.dt_own = real(dt)
        if self.conductive:
            m = (sig != 0) & (ieps != 0)
            tau = np.min((1 / ieps[m].astype(real)) / sig[m].astype(real))
            if self.dt_own > tau:
                self.dt_own = tau
        self.dt = float(self.dt_own)
        up = lambda a: torch.as_tensor(np.ascontiguousarray(a.transpose(2, 1, 0)), device=self.dev).reshape(-1)  # noqa: E731
        self.ieps, self.sig = up(ieps), up(sig)
        if block is not None:
            at = torch.as_tensor(np.flatnonzero(block.ravel(order="F")), device=self.dev)
            self.ieps = self.ieps.index_put((at,), 1.0 / (eps * EPS0))
            self.sig = self.sig.index_put((at,), sigma)
            self.conductive = True
        ax = lambda a, d: torch.as_tensor(a, device=self.dev).view([-1 if 2 - q == d else 1 for q in range(3)])  # noqa: E731
        area = lambda a, d: torch.as_tensor(np.ascontiguousarray(a.T), device=self.dev).view(  # noqa: E731
            [(nx, ny, nz)[2 - q] if 2 - q != d else 1 for q in range(3)])
        full = lambda t: t.expand(self.shape).reshape(-1)  # noqa: E731
        pec_like = ("pec", "pml")
        masks = [None] * 3
        if any(b in pec_like for b in low + high):
            for d in range(3):
                v = torch.ones(self.shape, dtype=torch.float64, device=self.dev)
                for a in range(3):
                    if a != d:
                        ix = [slice(None)] * 3
                        ix[2 - a] = 0
                        v[tuple(ix)] = 0.0 if low[a] in pec_like else 1.0
                        ix[2 - a] = -1
                        v[tuple(ix)] = 0.0 if high[a] in pec_like else 1.0
                masks[d] = v.reshape(-1)
        one = lambda d: 1.0 if masks[d] is None else masks[d]  # noqa: E731
        self.cE = [full(ax(L[d], d)) * one(d) for d in range(3)]
        self.cH = [full(ax(tL[d], d)) for d in range(3)]
        self.fH = [full(area(iA[d], d)) * (self.dt / MU0) for d in range(3)]
        self.fE = [full(area(itA[d], d)) * one(d) * self.dt * self.ieps for d in range(3)]
        zero = lambda: torch.zeros(self.N, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.E, self.H = [zero() for _ in range(3)], [zero() for _ in range(3)]
        self.J = [zero() for _ in range(3)] if self.conductive else None
        self.off = (1, nx, nx * ny)

    def flat(self, f):
        return torch.cat(f)

    def cell(self, x, y):
        return int(np.abs(self.x - x).argmin()), int(np.abs(self.y - y).argmin())

    def window(self, i, j):
        """Ez of the 3x3 lines around (i, j), x index outer."""
        v = self.E[2].view(self.shape)[:, j - 1:j + 2, i - 1:i + 2]
        return v.permute(2, 1, 0).reshape(9, -1)

    def ghosts(self):
        nz, ny, nx = self.shape
        last = [(slice(None), slice(None), nx - 1), (slice(None), ny - 1), (nz - 1,)]
        for a in range(3):
            self.E[a].view(self.shape)[last[a]] = 0.0
            for d in range(3):
                if d != a:
                    self.H[d].view(self.shape)[last[a]] = 0.0

    def _up(self, v, a):
        return torch.cat([v[self.off[a]:], v.new_zeros(self.off[a])])

    def _down(self, v, a):
        return torch.cat([v.new_zeros(self.off[a]), v[:-self.off[a]]])

    def step(self, line=None):
        """One step; ``line`` = (i, j, Jz along z)."""
        u = [self.E[d] * self.cE[d] for d in range(3)]
        up, down = self._up, self._down
        curl = (u[1] - up(u[1], 2) - u[2] + up(u[2], 1), up(u[0], 2) - u[0] + u[2] - up(u[2], 0),
                u[0] - up(u[0], 1) - u[1] + up(u[1], 0))
        self.H = [self.H[d] - self.fH[d] * curl[d] for d in range(3)]
        w = [self.H[d] * self.cH[d] for d in range(3)]
        curl = (down(w[1], 2) - w[1] - down(w[2], 1) + w[2], w[0] - down(w[0], 2) + down(w[2], 0) - w[2],
                down(w[0], 1) - w[0] - down(w[1], 0) + w[1])
        J = list(self.J) if self.J is not None else [0.0, 0.0, 0.0]
        if line is not None:
            i, j, val = line
            at = i + j * self.shape[2] + torch.arange(self.shape[0], device=self.dev) * self.off[2]
            jz = J[2] if self.J is not None else torch.zeros_like(self.E[2])
            J[2] = jz.index_put((at,), val)
        self.E = [self.E[d] + self.fE[d] * curl[d] - (self.dt * self.ieps * J[d]) for d in range(3)]
        if self.conductive:
            self.J = [self.sig * self.E[d] for d in range(3)]


def _beam_line(f, arg, n):
    """Jz of the bunch on the z line at step n (the time in the solver's own type)."""
    v = arg["beta"] * C
    ti = 8.548921333333334 * arg["sigmaz"] / v
    t = n * f.dt_own
    s = f.z - v * t
    s0 = f.z.min() - v * ti
    prof = 1 / np.sqrt(2 * np.pi * arg["sigmaz"] ** 2) * np.exp(-((s - s0) ** 2) / (2 * arg["sigmaz"] ** 2))
    i, j = f.cell(arg["xsource"], arg["ysource"])
    return i, j, torch.as_tensor(arg["q"] * v * prof / f.L[0][i] / f.L[1][j], device=f.dev)


def _wakesolve_exact(case, seed, steps=None):
    f = _Fit(case)
    arg = _beam_args(case, seed)
    v = arg["beta"] * C
    ti = 8.548921333333334 * arg["sigmaz"] / (np.sqrt(arg["beta"]) * v)
    if steps is None:
        wl = case["wakelength"]
        steps = int((wl + ti * v + (f.z.max() - f.z.min())) / v / f.dt_own)
    else:
        wl = (steps + 0.5) * f.dt * v - ti * v - (f.z.max() - f.z.min())
    i, j = f.cell(arg["xtest"], arg["ytest"])
    hist = torch.empty((9, case["nz"], steps), dtype=torch.float64, device=f.dev)
    for n in range(steps):
        hist[:, :, n] = f.window(i, j)
        f.step(line=_beam_line(f, arg, n))
    t = np.arange(0, steps * f.dt_own, f.dt_own)
    res = _wake_exact(hist, t, f.z, f.dz, f.x[i - 1:i + 2], f.y[j - 1:j + 2], wl, arg["sigmaz"], ti, arg["q"], 0, v)
    return res, f


def _samples(t, z, wl, ti, v, nt, skip):
    """The s axis, its step and, for each (s, z), the step of the history that is summed."""
    dt = t[2] - t[1]
    zmin = np.min(z)
    zz = z[skip:len(z) - skip]
    s = np.arange(-ti * v, wl, dt * v)
    it = ((((zz[None, :] + s[:, None]) / v - zmin / v) - t[0] + ti) / dt).astype(np.int64)
    ok = (it < nt) & (it >= -nt)
    return s, np.where(it < 0, it + nt, it), ok


def _bins(s, v, fmax):
    ds = np.mean(s[1:] - s[:-1])
    N = int((v / ds) // fmax * 1001)
    f = np.fft.fftfreq(N, ds / v)
    return ds, N, f, np.logical_and(f >= 0, f < fmax)


def _wake_exact(hist, t, z, dz, xf, yf, wl, sigmaz, ti, q, skip, v=C):
    nt = min(len(t), hist.shape[2])
    s, it, ok = _samples(t, z, wl, ti, v, nt, skip)
    dev = hist.device
    nz, ns = it.shape[1], len(s)
    idx = torch.as_tensor(np.where(ok, it, 0), device=dev).T.contiguous()
    keep = torch.as_tensor(ok.astype(np.float64), device=dev).T.contiguous()
    coef = torch.as_tensor(np.asarray(dz)[:nz], device=dev)[:, None]
    WP = np.empty((9, ns))
    prev = 0.0
    for w in range(9):
        part = (torch.gather(hist[w, skip:skip + nz], 1, idx) * keep * coef).sum(0).cpu().numpy()
        prev = (prev + part) / (q * 1e12)
        WP[w] = prev
    step = s[2] - s[1]
    prefix = lambda a: np.concatenate([[0.0], np.cumsum(a.astype(np.longdouble))[:-1].astype(np.float64)]) * step  # noqa: E731
    WPx = -(prefix(WP[7]) - prefix(WP[1])) / (xf[2] - xf[0])
    WPy = -(prefix(WP[5]) - prefix(WP[3])) / (yf[2] - yf[0])
    ds, N, f, m = _bins(s, v, v / (3.0 * sigmaz))
    lam = 1 / (sigmaz * np.sqrt(2 * np.pi)) * np.exp(-(s ** 2) / (2 * sigmaz ** 2))
    F = lambda a: np.fft.fft(a, n=N)[m] * ds  # noqa: E731
    lamf = F(lam * v)
    return {"WP": WP[4], "WPx": WPx, "WPy": WPy, "Z": -F(WP[4] * 1e12) / lamf,
            "Zx": 1j * F(WPx * 1e12) / lamf, "Zy": 1j * F(WPy * 1e12) / lamf}


def _adjoint_exact(case, seed):
    """Loss and gradient by torch's own differentiation of the steps, from checkpoints."""
    from torch.utils.checkpoint import checkpoint
    arg = _beam_args(case, seed)
    er, sg = (torch.tensor(a, device=_device(), requires_grad=True) for a in _params(case, seed))
    f = _Fit(case, eps=er, sigma=sg, block=_block(case))
    v, nt = arg["beta"] * C, case["steps"]
    ti = 8.548921333333334 * arg["sigmaz"] / (np.sqrt(arg["beta"]) * v)
    wl = (nt + 0.5) * f.dt * v - ti * v - (f.z.max() - f.z.min())
    i, j = f.cell(arg["xtest"], arg["ytest"])
    line = i + j * f.shape[2] + torch.arange(f.shape[0], device=f.dev) * f.off[2]

    def segment(a, b, *state):
        f.E, f.H, f.J = list(state[0:3]), list(state[3:6]), list(state[6:9])
        f.ieps, f.sig, f.fE = state[9], state[10], list(state[11:14])
        ez = []
        for n in range(a, b):
            ez.append(f.E[2][line])
            f.step(line=_beam_line(f, arg, n))
        return (torch.stack(ez, 1), *f.E, *f.H, *f.J)

    fixed = (f.ieps, f.sig, *f.fE)
    state, ez = (*f.E, *f.H, *f.J), []
    for a in range(0, nt, 25):
        out = checkpoint(segment, a, min(nt, a + 25), *state, *fixed, use_reentrant=False)
        ez.append(out[0])
        state = out[1:]
    hist = torch.cat(ez, 1)
    s = np.arange(-ti * v, wl, f.dt * v)
    it = ((((f.z[None, :] + s[:, None]) / v - f.z.min() / v) + ti) / f.dt).astype(np.int64)
    ok = (it < nt) & (it >= -nt)
    it = np.where(it < 0, it + nt, it)
    up = lambda a: torch.as_tensor(a, device=f.dev)  # noqa: E731
    vals = hist[torch.arange(case["nz"], device=f.dev)[None, :], up(np.where(ok, it, 0))]
    WP = (vals * up(ok.astype(np.float64)) * up(f.dz)[None, :]).sum(1) / (arg["q"] * 1e12)
    ds, N, freq, m = _bins(s, v, v / (3.0 * arg["sigmaz"]))
    keep = np.flatnonzero(m & (freq >= F_BAND[0]) & (freq <= F_BAND[1]))
    D = up(np.exp(-2j * np.pi * np.outer(keep, np.arange(len(s))) / N))
    lam = 1 / (arg["sigmaz"] * np.sqrt(2 * np.pi)) * np.exp(-(s ** 2) / (2 * arg["sigmaz"] ** 2))
    Z = -(D @ (WP * 1e12).to(torch.complex128)) / (D @ up(lam * v).to(torch.complex128))
    loss = torch.trapezoid(Z.real ** 2 + Z.imag ** 2, up(freq[keep]))
    ge, gs = torch.autograd.grad(loss, (er, sg))
    return {"loss": float(loss), "eps": ge.cpu().numpy(), "sigma": gs.cpu().numpy()}
