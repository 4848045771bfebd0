"""Calls at the edges of a kernel's or a rule's range, each against the general
path or the definition."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PEC = (["pec"] * 3, ["pec"] * 3)
OPEN = (["pec", "pec", "abc"], ["pec", "pec", "abc"])


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _solver(shape, bcs=PEC, dtype=np.float64, sigma=10.0, **kw):
    import wakis_b200 as wb
    g = wb.GridFIT3D(-0.03, 0.031, -0.02, 0.022, -0.04, 0.043, *shape, verbose=0)
    m = np.zeros(shape, bool)
    m[2:shape[0] // 2, 3:shape[1] // 2, 1:shape[2] // 2] = True
    g.add_solid("a", m, [4.0, 1.0, sigma])
    return wb.SolverFIT3D(g, bc_low=bcs[0], bc_high=bcs[1], dtype=dtype, bg=[1.0, 1.0],
                          use_stl=True, use_sibc=False, verbose=0, **kw)


def _random_state(s, e=True, seed=7):
    rng = np.random.default_rng(seed)
    s._first_step()
    if e:
        s.E.fromarray(300 * rng.standard_normal(3 * s.N))
    s.H.fromarray(rng.standard_normal(3 * s.N))


def _equal(a, b):
    return torch.equal(a.E.array, b.E.array) and torch.equal(a.H.array, b.H.array)


@pytest.mark.parametrize("dtype,shape", [(np.float32, (71, 21, 13)), (np.float32, (70, 33, 11)),
                                         (np.float32, (33, 35, 19)), (np.float64, (71, 21, 13)),
                                         (np.float64, (33, 35, 19))])
@pytest.mark.parametrize("tile", [(8, 1), (8, 2), (8, 5), (16, 3), (16, 64)])
def test_last_partial_row_group(dtype, shape, tile):
    """Closed grids whose 3 Ny Nz rows are no multiple of the group: the rows
    past the last whole group, filled in by hand on the top plane, wherever
    the chunks of planes end."""
    sol = []
    for kernel in ("auto", "twopass"):
        s = _solver(shape, dtype=dtype)
        s.kernel, s.tile, s.steps_per_launch = kernel, tile, 1
        _random_state(s)
        s._advance(6, 0)
        s.check_status()
        sol.append(s)
    assert _equal(*sol)


@pytest.mark.parametrize("dtype,shape", [(np.float64, (33, 24, 20)), (np.float64, (9, 8, 5)),
                                         (np.float32, (34, 24, 20)), (np.float32, (33, 17, 21)),
                                         (np.float64, (32, 24, 20)), (np.float32, (32, 17, 21))])
def test_two_steps_per_launch_on_any_row_length(dtype, shape):
    """steps_per_launch = 2 on closed, clean grids: rows that are no multiple
    of 16 bytes take one step per launch, the others pairs; the fields are the
    two-pass schedule's either way."""
    from wakis_b200.sources import Beam
    sol = []
    for kernel, spl in (("auto", 2), ("twopass", 1)):
        s = _solver(shape, dtype=dtype)
        s.kernel, s.steps_per_launch = kernel, spl
        bp = Beam(q=1e-9, sigmaz=0.005).params(s)
        s._advance(10, 0, beam=bp)
        s._advance(7, 10, beam=bp)
        s.check_status()
        sol.append(s)
    a, b = sol
    assert a._faces_clean and np.abs(a.E.numpy()).max() > 0
    assert _equal(a, b)


@pytest.mark.parametrize("ns,n_win", [(1, 1), (33, 9), (64, 3)])
@pytest.mark.parametrize("carry", [0, 1])
@pytest.mark.parametrize("q", [1e3, -1e3])
def test_wake_potential_of_no_z_cells_is_the_empty_sum(ns, n_win, carry, q):
    """nz = 0: every sample of every window is written, as 0 / q."""
    from wakis_b200 import _native
    f = lambda n: torch.ones(n, dtype=torch.float64, device="cuda")
    hist, z, s = f(n_win * 2 * 8), f(1), f(ns)
    win = torch.arange(n_win, dtype=torch.int32, device="cuda")
    order = torch.arange(8, dtype=torch.int64, device="cuda")
    WP = torch.full((n_win, ns), float("nan"), dtype=torch.float64, device="cuda")
    _native.check(_native.lib().wk_wake_potential(
        _ptr(hist), _native.WK_F64, 8, 2, _ptr(win), n_win, carry, _ptr(z), _ptr(z), 0, 0, _ptr(s),
        ns, _ptr(order), 8, 3e8, 0.0, 1.0, 0.0, 0.0, 1e-12, q, 0, _ptr(WP), _stream()),
        "wk_wake_potential")
    ref = np.empty((n_win, ns))
    acc = np.zeros(ns)
    for w in range(n_win):
        ref[w] = acc = (acc if carry else np.zeros(ns)) / q
    got = WP.cpu().numpy()
    assert np.array_equal(got, ref) and np.array_equal(np.signbit(got), np.signbit(ref))


@pytest.mark.parametrize("length,N,at", [(300, 700, 3), (300, 701, 257), (1000, 4001, 999), (40, 64, 0)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1.7e308])
def test_dft_bins_of_infinite_signals(length, N, at, value):
    """One infinite entry (or ones whose sum overflows) gives infinite parts
    where the term-by-term sum is infinite and NaN only where that sum is NaN;
    the signal beside it is not affected."""
    from wakis_b200 import _native
    rng = np.random.default_rng(at)
    x = rng.standard_normal((2, length))
    x[0, at] = value
    if np.isfinite(value):
        x[0, :] = value                       # bin 0 overflows
    nb = 6
    out = torch.empty((2, nb, 2), dtype=torch.float64, device="cuda")
    t = torch.as_tensor(x, device="cuda")
    _native.check(_native.lib().wk_dft_bins(_ptr(t), 2, length, N, nb, _ptr(out), _stream()),
                  "wk_dft_bins")
    got = out.cpu().numpy()
    assert np.isfinite(got[1]).all()
    if np.isfinite(value):
        assert got[0, 0, 0] == np.inf and got[0, 0, 1] == 0.0
        return
    for m in range(nb):
        # exact quarter turns decide where an infinite entry meets a zero
        r = (m * at) % N
        turn = 2 * np.pi * r / N
        c = 0.0 if 4 * r in (N, 3 * N) else np.cos(turn)
        s = 0.0 if 2 * r in (0, N) else np.sin(turn)
        for part, f in ((0, c), (1, -s)):
            want = value * f if f != 0 and not np.isnan(value) else np.nan
            assert np.array_equal(got[0, m, part], want, equal_nan=True), (m, part)


@pytest.mark.parametrize("nz", [1, 2])
def test_wake_potential_of_a_history_past_int_columns(nz):
    """More than 2^31 columns (FP32, 8.6 GB a row): the entries of the last
    ones are the ones read."""
    from wakis_b200 import _native
    nt, rows, ns, dt = 2 ** 31 + 9, nz, 8 - nz + 1, 1e-12
    hist = torch.empty(rows * nt, dtype=torch.float32, device="cuda")
    order = torch.arange(nt - 8, nt, dtype=torch.int64, device="cuda")
    rng = np.random.default_rng(1)
    vals = rng.standard_normal((rows, 8)).astype(np.float32)
    for r in range(rows):
        hist[r * nt + nt - 8:(r + 1) * nt] = torch.as_tensor(vals[r], device="cuda")
        hist[r * nt:r * nt + 8] = float("nan")
    v = 1.0 / dt                              # column = z + s in units of one
    f = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")
    z, dz, s = f(np.arange(nz) + 0.0), f(np.ones(nz)), f(np.arange(ns) + 0.25)
    WP = torch.full((1, ns), float("nan"), dtype=torch.float64, device="cuda")
    win = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.check(_native.lib().wk_wake_potential(
        _ptr(hist), _native.WK_F32, nt, rows, _ptr(win), 1, 0, _ptr(z), _ptr(dz), nz, 0, _ptr(s),
        ns, _ptr(order), 8, v, 0.0, 1.0, 0.0, 0.0, dt, 1.0, 0, _ptr(WP), _stream()),
        "wk_wake_potential")
    ref = np.zeros(ns)
    for k in range(nz):
        ref += vals[k, np.arange(ns) + k].astype(np.float64)
    assert np.array_equal(WP.cpu().numpy()[0], ref)
    del hist
    torch.cuda.empty_cache()


@pytest.mark.parametrize("ns", [65535, 65536, 65537, 131073, 200003])
def test_transverse_prefix_sums_of_long_axes(ns):
    """Axes on both sides of 128 * 2^9 samples, where another kernel takes them:
    numpy's sums value for value."""
    from wakis_b200 import _native
    rng = np.random.default_rng(ns)
    WP = rng.standard_normal((9, ns))
    t = torch.as_tensor(WP, device="cuda")
    wx, wy = (torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(2))
    ds, dx, dy = 1e-3, 2e-3, 3e-3
    _native.check(_native.lib().wk_trans_wake(_ptr(t), ns, ds, dx, dy, _ptr(wx), _ptr(wy), _stream()),
                  "wk_trans_wake")
    wx, wy = wx.cpu().numpy(), wy.cpu().numpy()
    for n in sorted(set(rng.integers(0, ns, 100).tolist()) | {0, 1, 129, 65534, ns - 1}):
        i = {w: np.sum(WP[w, 0:n]) * ds for w in (7, 1, 5, 3)}
        assert wx[n] == -(i[7] - i[1]) / dx and wy[n] == -(i[5] - i[3]) / dy


@pytest.fixture
def few_sms():
    """A stream of a context that has a part of the device's SMs."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        if int(r[0]) != 0:
            pytest.skip(f"no partition of the SMs here ({r[0]})")
        return r[1] if len(r) == 2 else r[1:]

    torch.zeros(1, device="cuda")
    dev = ok(drv.cuDeviceGet(torch.cuda.current_device()))
    sm = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, _, _ = ok(drv.cuDevSmResourceSplitByCount(1, sm, 0, 16))
    desc = ok(drv.cuDevResourceGenerateDesc(parts, 1))
    ctx = ok(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(drv.cuGreenCtxStreamCreate(
        ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(stream))
    torch.cuda.synchronize()
    drv.cuStreamDestroy(stream)
    drv.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("precision", ["float64", "float32", "fp32c"])
def test_small_grids_on_a_part_of_the_sms(few_sms, precision):
    """Where the launch of all steps is refused for want of resident blocks, the
    call runs step by step: the fields of the other path."""
    kw = {"precision": "fp32c"} if precision == "fp32c" else {"dtype": np.dtype(precision).type}
    sol = []
    for stream in (few_sms, torch.cuda.current_stream()):
        s = _solver((44, 33, 57), bcs=OPEN, **kw)
        s._desc.wait_ns = 200_000_000
        _random_state(s, e=precision != "fp32c")
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            s._advance(9, 0)
            s.check_status()
        torch.cuda.synchronize()
        sol.append(s)
    assert _equal(*sol)
    assert int(sol[0]._sync.abs().sum().item()) == 0


def _cavities(n, precision, shape=(16, 20, 24)):
    import wakis_b200 as wb
    sol = []
    for q in range(n):
        g = wb.GridFIT3D(-0.008, 0.008, -0.01, 0.01, -0.012, 0.012, *shape, verbose=0)
        m = np.ones(shape, bool)
        m[3:13, 4:16, :] = False
        g.add_solid("wall", m, [1.0, 1.0, 0.5 + 0.05 * q])
        w = wb.WakeSolver(q=1e-9, sigmaz=3e-3, save=False, verbose=0)
        kw = {"precision": "fp32c"} if precision == "fp32c" else {"dtype": np.dtype(precision).type}
        sol.append(wb.SolverFIT3D(g, w, bc_low=OPEN[0], bc_high=OPEN[1], use_stl=True, use_sibc=False,
                                  bg="vacuum", verbose=0, **kw))
    return sol


@pytest.mark.parametrize("precision,count,form", [("fp32c", 2, "loop"), ("fp32c", 14, "batched"),
                                                  ("float64", 2, "loop"), ("float64", 6, "graph"),
                                                  ("float32", 6, "graph")])
def test_batch_form_by_count_and_its_results(precision, count, form):
    """The form that is picked, and the wake potentials of single runs whose
    steps are launched one by one."""
    from wakis_b200 import batch
    sol = _cavities(count, precision)
    b = batch.BatchedWakeSolve(sol, 251, tune=False)
    assert b.launch == form
    b.run()
    ref = _cavities(count, precision)
    for s, r in zip(sol, ref):
        r.steps_per_launch = 1
        r.wakesolve(wakelength=batch.BatchedWakeSolve.wakelength_for(r, 251))
        assert np.abs(r.wake.WP).max() > 0
        assert np.array_equal(s.wake.WP_3d, r.wake.WP_3d) and np.array_equal(s.wake.Zx, r.wake.Zx)


@pytest.mark.parametrize("precision", [None, "fp32c"])
@pytest.mark.parametrize("tune", [False, True])
def test_graph_of_per_instance_launches(precision, tune):
    """launch='graph': uneven pillboxes (surface impedance walls among them) on
    several streams, the step index from the device counter, an odd and an even
    number of steps after the first; the results of single runs whose steps are
    launched one by one."""
    from wakis_b200 import batch

    def boxes():
        return [batch.build_pillbox(cell=2e-3, precision=precision, **q)[2] for q in (
            dict(R=0.020, L=0.030, beta=0.9, sigma=1e4), dict(R=0.026, L=0.036, beta=0.6, sigma=3e5),
            dict(R=0.022, L=0.040, beta=1.0, sigma=2e3))]

    for steps in (600, 601):
        inst, solo = boxes(), boxes()
        b = batch.BatchedWakeSolve(inst, steps, launch="graph", streams=4, tune=tune)
        assert b.launch == "graph"
        b.run()
        for s, r in zip(inst, solo):
            r.steps_per_launch = 1
            r.wakesolve(wakelength=batch.BatchedWakeSolve.wakelength_for(r, steps))
            assert r.Nt == steps and np.abs(r.wake.WP).max() > 0
            assert np.array_equal(s.wake.WP, r.wake.WP) and np.array_equal(s.wake.Z, r.wake.Z)
            assert np.array_equal(s.E.numpy(), r.E.numpy())


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,shape", [(80, (12, 10, 90)), (290, (9, 8, 300))])
def test_one_launch_with_many_materials(dtype, n, shape):
    """More materials than fit beside the tiles (ids of one and two bytes)."""
    import wakis_b200 as wb
    from wakis_b200 import _native
    sol = []
    for kernel in ("auto", "cell"):
        g = wb.GridFIT3D(-0.03, 0.031, -0.02, 0.022, -0.14, 0.143, *shape, verbose=0)
        for q in range(n):
            m = np.zeros(shape, bool)
            m[2:8, 2:7, 4 + q] = True
            g.add_solid(f"m{q}", m, [1.0 + 0.01 * q, 1.0, 0.1 * (q % 7)])
        s = wb.SolverFIT3D(g, bc_low=OPEN[0], bc_high=OPEN[1], dtype=dtype, bg=[1.0, 1.0],
                           use_stl=True, use_sibc=False, verbose=0)
        s.kernel = kernel
        assert s._desc.n_mat > (64 if n < 256 else 256)
        _random_state(s)
        if kernel == "auto":
            assert _native.lib().wk_fit_one_launch(s._step_desc(), 9) == 1
        s._advance(9, 0)
        s.check_status()
        sol.append(s)
    assert _equal(*sol)


@pytest.mark.parametrize("precision", ["float64", "float32", "fp32c"])
def test_one_launch_that_gives_up(precision):
    """Waits without time: the blocks leave, the host sees the status, the
    barrier words are zero again and the next run is a run of its own."""
    kw = {"precision": "fp32c"} if precision == "fp32c" else {"dtype": np.dtype(precision).type}
    a, b = (_solver((36, 33, 57), bcs=OPEN, **kw) for _ in range(2))
    _random_state(a, e=False)
    a._desc.wait_ns = -1
    a._advance(9, 0)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        a.check_status()
    assert int(a._sync.abs().sum().item()) == 0
    a._desc.wait_ns = 0
    for s in (a, b):
        s.reset_fields()
        s.step_0, s.nstep = True, 0
        _random_state(s, e=False)
        s._advance(9, 0)
        s.check_status()
    assert _equal(a, b) and np.abs(a.E.numpy()).max() > 0


@pytest.mark.parametrize("precision", ["float64", "float32", "fp32c"])
@pytest.mark.parametrize("shape,bcs", [((36, 33, 57), OPEN), ((33, 20, 41), PEC), ((37, 21, 40), OPEN)])
def test_one_launch_calls_between_single_steps(precision, shape, bcs):
    """Calls that run in one launch, single steps and host traffic in turn: what
    one leaves in either buffer is what the next one needs."""
    kw = {"precision": "fp32c"} if precision == "fp32c" else {"dtype": np.dtype(precision).type}
    sol, out = [], []
    for spl in (0, 1):
        s = _solver(shape, bcs=bcs, **kw)
        s.steps_per_launch = spl
        _random_state(s, e=False)
        rng = np.random.default_rng(5)
        ez = []
        for n in (9, 1, 8, 3, 1, 1, 12):
            s._advance(n, s.nstep)
            lines = 1e-3 * rng.standard_normal((7, s.Nz))
            buf = torch.empty((7, 9, s.Nz), dtype=s._cap_dtype).pin_memory()
            s.run_with_io(torch.as_tensor(lines).to(s._cap_dtype).pin_memory(), buf)
            ez.append(buf.clone())
        s.check_status()
        sol.append(s)
        out.append(ez)
    assert _equal(*sol) and all(torch.equal(a, b) for a, b in zip(*out))
    assert np.abs(sol[0].E.numpy()).max() > 0
