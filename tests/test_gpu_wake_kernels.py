"""The wake kernels at the edges of their work splits, against numpy."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

C = 299792458.0


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _dev(a, dtype=np.float64):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=dtype), device="cuda")


@pytest.mark.parametrize("nz,ns,n_win", [(1, 1, 9), (15, 33, 9), (16, 40, 1), (17, 64, 9), (63, 31, 9),
                                         (64, 65, 9), (65, 7, 9), (1024, 33, 3), (1025, 33, 3)])
@pytest.mark.parametrize("counter", [0, 1])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_wake_potential_equals_sequential_sums(nz, ns, n_win, counter, dtype):
    """WP_3d value for value in upstream's order (z, then window, carried over),
    with columns that fall outside the history."""
    from wakis_b200 import _native
    lib = _native.lib()
    rng = np.random.default_rng(nz + ns)
    dt, dz0, ti = 1e-12, 1e-3, 5e-12
    nt = ns + 2 * nz
    z = (np.arange(nz) + 0.5) * dz0
    dz = dz0 * (1 + 0.1 * rng.random(nz))
    s = np.arange(ns) * dt * C - ti * C
    hist = rng.standard_normal((n_win, nz + 2, nt)).astype(dtype)
    order = rng.permutation(nt).astype(np.int64)
    out = {}
    for carry in (0, 1):
        WP = torch.zeros((n_win, ns), dtype=torch.float64, device="cuda")
        args = [_dev(hist, dtype), _dev(np.arange(n_win), np.int32), _dev(z), _dev(dz), _dev(s),
                _dev(order, np.int64)]
        h, win, zt, dzt, st, ot = args
        code = _native.WK_F64 if dtype == np.float64 else _native.WK_F32
        _native.check(lib.wk_wake_potential(
            _ptr(h), code, nt, nz + 2, _ptr(win), n_win, carry, _ptr(zt), _ptr(dzt), nz, 1, _ptr(st),
            ns, _ptr(ot), nt - 3, C, z.min(), z.max(), 0.0, ti, dt, 1e3, counter, _ptr(WP),
            _stream()), "wk_wake_potential")
        ref = np.empty((n_win, ns))
        prev = np.zeros(ns)
        for w in range(n_win):
            acc = prev.copy() if carry else np.zeros(ns)
            for k in range(nz):
                if counter:
                    ts = (z[nz - 1 - k] - s) / -C - z.max() / -C - 0.0 + ti
                    row, coef = nz - 1 - k + 1, -dz[k]
                else:
                    ts = (z[k] + s) / C - z.min() / C - 0.0 + ti
                    row, coef = k + 1, dz[k]
                it = (ts / dt).astype(np.int64)
                ok = it < nt - 3
                it = np.where(it < 0, it + nt - 3, it)
                ok &= it >= 0
                e = hist[w, row, order[np.where(ok, it, 0)]].astype(np.float64)
                acc = np.where(ok, acc + e * coef, acc)
            ref[w] = prev = acc / 1e3
        out[carry] = WP.cpu().numpy(), ref
    for a, b in out.values():
        assert np.array_equal(a, b)


@pytest.mark.parametrize("ns", [1, 2, 7, 9, 127, 130, 257, 1025, 4097, 4111, 8200])
def test_transverse_prefix_sums_are_numpys(ns):
    """WPx, WPy from numpy's own pairwise sums, value for value."""
    from wakis_b200 import _native
    rng = np.random.default_rng(ns)
    WP = rng.standard_normal((9, ns))
    t = _dev(WP)
    wx, wy = (torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(2))
    ds, dx, dy = 1e-3, 2e-3, 3e-3
    _native.check(_native.lib().wk_trans_wake(_ptr(t), ns, ds, dx, dy, _ptr(wx), _ptr(wy), _stream()),
                  "wk_trans_wake")
    pick = range(ns) if ns < 300 else sorted(set(rng.integers(0, ns, 200)) | {ns - 1})
    for n in pick:
        i = {w: np.sum(WP[w, 0:n]) * ds for w in (7, 1, 5, 3)}
        assert wx[n].item() == -(i[7] - i[1]) / dx
        assert wy[n].item() == -(i[5] - i[3]) / dy


@pytest.mark.parametrize("length,N,nbins,nsig", [(1, 1, 1, 1), (255, 300, 7, 2), (256, 256, 256, 3),
                                                 (257, 4001, 11, 1), (70000, 90001, 5, 2)])
def test_dft_bins_against_extended_precision(length, N, nbins, nsig):
    """The kept bins against numpy's transform in extended precision.  Bound:
    len / 256 + 2 fused adds of a thread, two roundings of the unit's product
    and of the unit itself, eight levels of the tree, each half an ulp of at
    most the sum of |x|."""
    from wakis_b200 import _native
    rng = np.random.default_rng(length)
    x = rng.standard_normal((nsig, length))
    out = torch.empty((nsig, nbins, 2), dtype=torch.float64, device="cuda")
    t = _dev(x)
    _native.check(_native.lib().wk_dft_bins(_ptr(t), nsig, length, N, nbins, _ptr(out), _stream()),
                  "wk_dft_bins")
    got = torch.view_as_complex(out).cpu().numpy()
    ref = np.fft.fft(x.astype(np.longdouble), n=N)[:, :nbins]
    bound = (length / 256 + 16) * 2.0 ** -52 * np.abs(x).sum(axis=1)
    assert np.all(np.abs((got - ref).astype(np.complex128)) <= bound[:, None])
