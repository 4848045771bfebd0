"""The rule that picks the launch form of a batch, on stand-ins for solvers."""

from types import SimpleNamespace

import pytest

pytest.importorskip("torch")

from wakis_b200 import _native, batch


class _Solver(SimpleNamespace):
    def _step_desc(self):
        return self._desc


def _solvers(n, shape, precision, closed=False, device="cuda:0"):
    d = SimpleNamespace(id_bytes=1, has_pec=1, has_pmc=0, pec_face=[0, 0, 0, 0] + [int(not closed)] * 2,
                        dtype={"fp32c": _native.WK_F32C, "float64": _native.WK_F64,
                               "float32": _native.WK_F32}[precision])
    return [_Solver(Nx=shape[0], Ny=shape[1], Nz=shape[2], precision=precision, device=device,
                    use_conductivity=True, _desc=d) for _ in range(n)]


TINY, MID, ODD = (16, 16, 32), (40, 40, 80), (33, 36, 61)


@pytest.mark.parametrize("precision,shape,closed,most", [
    ("fp32c", TINY, False, 12), ("fp32c", TINY, True, 12), ("fp32c", MID, False, 24),
    ("fp32c", MID, True, 8), ("fp32c", (17, 17, 32), False, 8), ("fp32c", ODD, False, None),
    ("float64", TINY, False, 4), ("float64", MID, False, 4), ("float64", MID, True, 2),
    ("float64", ODD, True, 8), ("float32", (34, 36, 61), False, 8), ("float32", (36, 36, 61), False, 4),
    ("float32", (25, 24, 48), False, 4)])
def test_form_by_the_count_of_instances(monkeypatch, precision, shape, closed, most):
    """Few instances run one after another, more are stepped together."""
    lib = SimpleNamespace(wk_fit_one_launch=lambda d, n: 1)
    monkeypatch.setattr(_native, "lib", lambda: lib)
    together = "batched" if precision == "fp32c" and shape[0] % 4 == 0 else "graph"
    for n in (1, 2, 3, 4, 5, 8, 9, 12, 13, 24, 25, 64):
        b = batch.BatchedWakeSolve(_solvers(n, shape, precision, closed), 100)
        assert b.launch == ("loop" if most is None or n <= most else together), n


def test_instances_of_several_devices_are_not_run_in_turn(monkeypatch):
    lib = SimpleNamespace(wk_fit_one_launch=lambda d, n: 1)
    monkeypatch.setattr(_native, "lib", lambda: lib)
    mixed = _solvers(1, MID, "float64") + _solvers(1, MID, "float64", device="cuda:1")
    assert not batch.loop_ok(mixed, 99)
    assert batch.loop_ok(mixed[:1], 99)
