"""Gauss-Jordan panel widths that negf_device_selected_inverse takes besides 8,
16 and 32: odd ones, ones wider than the update kernel's buffer, and ones as wide
as the block.

Tolerance: two backward-stable inversions differ by no more than n u cond, with
n the order of the whole matrix and u = 2^-53."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(negf, dev, npl, b, method, gj_nb, mixed=False, gj_update=0):
    from libnegf_b200._lib import c_double_p, int_array
    E = np.array([0.05, -0.3])
    o = negf.make_opts(eta=5e-2, gj_nb=gj_nb, precision="mixed" if mixed else "fp64", gj_update=gj_update)
    gd = np.empty(2 * npl * b * b, complex)
    rc = negf.load().negf_device_selected_inverse(
        dev.handle, 2, E.ctypes.data_as(c_double_p), ctypes.byref(o), method, 1 if method == 1 else 0,
        int_array([1]) if method == 1 else None, gd.ctypes.data, None, None, 0, None)
    return rc, E, gd.reshape(2, npl, b, b).transpose(0, 1, 3, 2)


def _device(negf, npl, b):
    rng = np.random.default_rng(b)
    cn = lambda: (rng.standard_normal((b, b)) + 1j * rng.standard_normal((b, b))) / np.sqrt(2 * b)
    Hd = [(a + a.conj().T) / 2 for a in (cn() for _ in range(npl))]
    Hu = [0.5 * cn() for _ in range(npl - 1)]
    s = -0.05j * np.eye(b)
    return negf.Device(Hd, Hu, s, s), Hd, Hu, s


@pytest.mark.parametrize("b", [113, 119, 130, 256])
@pytest.mark.parametrize("method", [0, 1])
def test_widths(negf, b, method):
    npl = 4  # two separators, two interiors of one layer
    dev, Hd, Hu, s = _device(negf, npl, b)
    ref = None
    for gj_nb in (0, 3, 8, 12, 20, 32, 33, 37, 48, 64, 120, 256):
        if gj_nb > 48 and b == 256 or gj_nb > 119 and b > 119:
            continue  # refused: see below
        rc, E, gd = _run(negf, dev, npl, b, method, gj_nb)
        assert rc == 0, gj_nb
        if ref is None:
            ref, bound = [], []
            for e in E:
                M = (e + 5e-2j) * np.eye(npl * b)
                for i in range(npl):
                    M[i * b:(i + 1) * b, i * b:(i + 1) * b] -= Hd[i] + (s if i == 0 else 0) + (s if i == npl - 1 else 0)
                    if i + 1 < npl:
                        M[i * b:(i + 1) * b, (i + 1) * b:(i + 2) * b] = -Hu[i]
                        M[(i + 1) * b:(i + 2) * b, i * b:(i + 1) * b] = -Hu[i].conj().T
                X = np.linalg.inv(M)
                ref.append([X[i * b:(i + 1) * b, i * b:(i + 1) * b] for i in range(npl)])
                bound.append(2.0 ** -53 * npl * b * np.linalg.cond(M) * np.linalg.norm(X))
        for g, r, t in zip(gd, ref, bound):
            assert max(np.linalg.norm(x - y) for x, y in zip(g, r)) <= t, gj_nb


@pytest.mark.parametrize("b,gj_nb", [(256, 64), (300, 48), (512, 32), (120, 120)])
def test_too_wide_is_refused(negf, b, gj_nb):
    from libnegf_b200._lib import NEGF_ERR_INVALID
    dev = _device(negf, 3, b)[0]
    for method in (0, 1):
        assert _run(negf, dev, 3, b, method, gj_nb)[0] == NEGF_ERR_INVALID


def test_int8_updates(negf):
    dev = _device(negf, 3, 130)[0]
    a = _run(negf, dev, 3, 130, 0, 0, mixed=True, gj_update=2)
    c = _run(negf, dev, 3, 130, 0, 48, mixed=True, gj_update=2)
    assert a[0] == 0 and c[0] == 0
    assert np.linalg.norm(a[2] - c[2]) <= 1e-10 * np.linalg.norm(a[2])
