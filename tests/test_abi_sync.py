"""The grid-barrier words of the step descriptor are checked before a launch."""

import ctypes
import os

import pytest

from wakis_b200 import _native


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(_native.LIB_PATH):
        from wakis_b200 import build
        build.build(verbose=False)
    return _native.lib()


def _desc():
    """A descriptor that passes the checks; its addresses are never read."""
    d = _native.FitDesc()
    d.Nx, d.Ny, d.Nz = 8, 9, 10
    for n in ("E", "H"):
        getattr(d, n)[0], getattr(d, n)[1] = 1 << 20, 1 << 21
    for n in ("mat_id", "mat_table", "Lx", "Ly", "Lz", "tLx", "tLy", "tLz", "iAx", "iAy", "iAz",
              "itAx", "itAy", "itAz"):
        setattr(d, n, 1 << 22)
    d.id_bytes, d.n_mat, d.dtype = 1, 1, _native.WK_F64
    return d


@pytest.mark.parametrize("sync,bad", [(None, False), (1 << 23, False), ((1 << 23) + 4, False),
                                      ((1 << 23) + 1, True), ((1 << 23) + 2, True)])
def test_sync_words_are_aligned(lib, sync, bad):
    """No steps, so that nothing is launched (without a device the call may end
    in its error instead of 0)."""
    d = _desc()
    d.sync = sync
    rc = lib.wk_fit_step(ctypes.byref(d), 0, 0, None)
    assert rc == 4 if bad else rc <= 0
    if bad:
        assert b"sync" in lib.wk_last_error()
