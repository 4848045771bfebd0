"""WakeSolver.solve and its steps on the host, the device kernels replaced by
torch expressions: a replaced step is run, and a step that fails leaves the
results of the steps before it."""

import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from wakis_b200.wakeSolver import WakeSolver

NS, NB = 12, 5


def _wake(cls=WakeSolver):
    """A solver with a history and stand-ins for the kernels."""
    w = cls(wakelength=1.0, sigmaz=0.1, save=False, verbose=0)
    w.set_history(torch.zeros((9, 4, 40), dtype=torch.float64), 40)
    s = np.linspace(-0.5, 0.6, NS)
    rng = np.random.default_rng(3)
    WP, WPxy = rng.standard_normal((9, NS)), rng.standard_normal((2, NS))

    def _wp(self, n_win, carry):
        self.s = s
        return torch.tensor(WP)

    def _bins(self, signals, samples, fmax):
        return self._dft(torch.stack([torch.as_tensor(x, dtype=torch.float64) for x in signals]),
                         samples, fmax)

    def _dft(self, x, samples, fmax):
        X = torch.fft.fft(x.to(torch.complex128), dim=-1)[:, :NB]
        return 0.1, np.arange(NB) * 1e9, X

    def _trans(self, WP3d, scan=False):
        return torch.tensor(WPxy)

    w._axis = lambda: (40, 1e-12, 0.0, 1.0, np.zeros(4), s)
    for f in (_wp, _bins, _dft, _trans):
        setattr(w, f.__name__, types.MethodType(f, w))
    return w, WP, WPxy


NAMES = ("WP", "WP_3d", "WPx", "WPy", "Z", "Zx", "Zy", "f", "lambdaf")


def _stepwise():
    w, WP, WPxy = _wake()
    for n in ("calc_long_WP_3d", "calc_trans_WP", "calc_long_Z", "calc_trans_Z"):
        getattr(w, n)()
    return w


def test_solve_equals_its_steps():
    w, WP, WPxy = _wake()
    w.solve()
    ref = _stepwise()
    for n in NAMES:
        assert np.allclose(getattr(w, n), getattr(ref, n), rtol=1e-14, atol=0), n


@pytest.mark.parametrize("name", ["calc_long_WP_3d", "calc_trans_WP", "calc_lambdas_analytic",
                                  "calc_long_Z", "calc_trans_Z"])
@pytest.mark.parametrize("how", ["subclass", "instance", "class"])
def test_a_replaced_step_is_run(name, how, monkeypatch):
    calls = []
    orig = getattr(WakeSolver, name)

    def step(self, **kw):
        calls.append(name)
        orig(self, **kw)

    cls = type("Own", (WakeSolver,), {name: step}) if how == "subclass" else WakeSolver
    w, WP, WPxy = _wake(cls)
    if how == "instance":
        setattr(w, name, types.MethodType(step, w))
    elif how == "class":
        monkeypatch.setattr(WakeSolver, name, step)
    w.solve()
    assert calls == [name]
    ref = _stepwise()
    for n in NAMES:
        assert np.allclose(getattr(w, n), getattr(ref, n), rtol=1e-14, atol=0), n


@pytest.mark.parametrize("fails,kept", [("_trans", ["WP", "WP_3d"]),
                                        ("_dft", ["WP", "WP_3d", "WPx", "WPy"]), ("_wp", [])])
def test_a_step_that_fails_leaves_the_results_before_it(fails, kept):
    """A second solve whose transverse integration or DFT raises (a range of
    frequencies without bins, say): the error, the new results of the steps
    before it, the earlier ones of the steps after it, the line density as
    given."""
    w, WP, WPxy = _wake()
    for n in NAMES:
        setattr(w, n, "earlier")

    def bad(self, *a, **k):
        raise ZeroDivisionError("no bins")

    setattr(w, fails, types.MethodType(bad, w))
    with pytest.raises(ZeroDivisionError):
        w.solve()
    ref = _stepwise()
    for n in NAMES:
        if n in kept:
            assert np.array_equal(getattr(w, n), getattr(ref, n)), n
        else:
            assert getattr(w, n) == "earlier", n
    assert (w.lambdas is None) == (fails != "_dft")


def test_a_line_density_that_cannot_be_scaled_is_refused():
    w, WP, WPxy = _wake()
    w.lambdas = [0.0] * NS
    with pytest.raises(TypeError):
        w.solve()
    assert np.array_equal(w.WPx, WPxy[0]) and w.Z is None
