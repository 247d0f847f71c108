"""NaN and infinities never come back as a success with finite numbers."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAD = {"nan": complex(np.nan, 0.0), "nan_im": complex(0.0, np.nan), "inf_inf": complex(np.inf, -np.inf),
       "inf_nan": complex(np.inf, np.nan)}


def _mat(rng, n):
    return rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))


def _device(negf, npl, b):
    rng = np.random.default_rng(npl * b)
    Hd, Hu = [], []
    for _ in range(npl):
        A = _mat(rng, b) / np.sqrt(2 * b)
        Hd.append((A + A.conj().T) / 2)
    for _ in range(npl - 1):
        Hu.append(0.25 * _mat(rng, b) / np.sqrt(b))
    s = -0.05j * np.eye(b)
    return negf.Device(Hd, Hu, s, s)


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("n", [1, 20, 33, 70, 150])
def test_unpivoted_lu(negf, n, bad):
    """A non-finite pivot reaches every element of the block's inverse."""
    from libnegf_b200._lib import ptr_array
    rng = np.random.default_rng(n)
    for i, j in {(0, 0), (n // 2, n // 2), (n - 1, n - 1), (n - 1, 0)}:
        a = _mat(rng, n) + 3.0 * n * np.eye(n)
        a[i, j] = BAD[bad]
        d, fill = negf.to_device(a), (ctypes.c_uint8 * 1)()
        rc = negf.load().negf_selected_inverse_batched(1, 1, n, ptr_array([d.data_ptr()]), fill, 3, 0, 0, None)
        assert rc != 0 or np.isnan(negf.to_host(d)).all()


@pytest.mark.parametrize("npl,b", [(3, 24), (3, 70)])
def test_selected_inverse_nan_energy(negf, npl, b):
    """The energies beside a NaN are not touched by it."""
    d = _device(negf, npl, b)
    alone = d.selected_inverse([0.1], "selinv", eta=1e-2)
    both = d.selected_inverse([0.1, np.nan], "selinv", eta=1e-2)
    for x, y in zip(alone, both):
        assert all(np.array_equal(p, q) for p, q in zip(x[0], y[0]))
        assert all(np.isnan(q).all() for q in y[1])


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("n", [1, 8, 40, 100, 140, 300, 520])
def test_inversion(negf, n, bad):
    """The Gauss-Jordan kernels report a matrix whose rows turn into NaN: NaN
    rows are never pivots, so a later column has no candidate left."""
    from libnegf_b200._lib import NEGF_ERR_SINGULAR, int_array, ptr_array
    rng = np.random.default_rng(n)
    good = _mat(rng, n)
    for i, j in {(0, 0), (n // 2, n // 2), (n - 1, 0), (0, n - 1)}:
        a = good.copy()
        a[i, j] = BAD[bad]
        dA, dO = [negf.to_device(x) for x in (good, a)], [negf.dzeros(n, n) for _ in range(2)]
        info = (ctypes.c_int32 * 2)()
        rc = negf.load().negf_zinv_batched(2, int_array([n, n]), ptr_array([x.data_ptr() for x in dA]), int_array([n, n]),
                                           ptr_array([x.data_ptr() for x in dO]), int_array([n, n]), info, None)
        assert info[0] == 0
        if n > 1:
            assert rc == NEGF_ERR_SINGULAR and info[1] > 0
        else:
            assert rc == NEGF_ERR_SINGULAR or np.isnan(negf.to_host(dO[1])).all()


@pytest.mark.parametrize("bad", sorted(BAD) + ["inf"])
@pytest.mark.parametrize("ops", ["NN", "TC", "CT"])
@pytest.mark.parametrize("k", [20, 130, 300, 600])
def test_mixed_product(negf, ops, k, bad):
    """A bad element of op(A) or op(B) makes its row or column of the result NaN
    and leaves the rest to the last bit."""
    rng = np.random.default_rng(k)
    m, n = 70, 45
    v = BAD.get(bad, complex(-np.inf, 1.0))
    op = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
    A, B, C = _mat(rng, k)[:m].copy() if k >= m else _mat(rng, m)[:, :k].copy(), _mat(rng, max(k, n))[:k, :n].copy(), \
        _mat(rng, m)[:, :n].copy()

    def run(a, b):
        out = negf.to_device(C.copy())
        negf.be_gemm_batched_(ops[0], ops[1], [(1.0 - 0.5j, negf.to_device(np.ascontiguousarray(op[ops[0]](a))),
                                                negf.to_device(np.ascontiguousarray(op[ops[1]](b))), 1.0, out)], "mixed")
        return negf.to_host(out)

    clean = run(A, B)
    assert np.isfinite(clean).all()
    for i in (0, 33, m - 1):
        X = A.copy()
        X[i, k // 2] = v
        got = run(X, B)
        rest = np.arange(m) != i
        assert np.isnan(got[i]).all() and np.array_equal(got[rest], clean[rest])
    for j in (0, 17, n - 1):
        Y = B.copy()
        Y[k - 1, j] = v
        got = run(A, Y)
        rest = np.arange(n) != j
        assert np.isnan(got[:, j]).all() and np.array_equal(got[:, rest], clean[:, rest])


def test_mixed_selected_inverse_nan_energy(negf):
    d = _device(negf, 3, 130)
    r = d.selected_inverse([0.1, np.nan], "selinv", "mixed", eta=1e-2)
    for x in r:
        assert all(np.isfinite(q).all() for q in x[0]) and all(np.isnan(q).all() for q in x[1])
