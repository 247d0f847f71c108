"""Unpivoted LU with both triangular inverses (32-blocks, joins of 32, 64, ..) and
the triangular inverses behind be_trsm! / be_getri!, at sizes around the block
edges, against numpy.

Tolerance: products of explicit triangular inverses of diagonally dominant
blocks, condition below 10: n u times a factor 100 for the chain of products."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mat(rng, n):
    return rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n * np.eye(n)


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [1, 5, 31, 32, 33, 63, 64, 65, 96, 100, 129, 257])
@pytest.mark.parametrize("nsys", [1, 3])
def test_selected_inverse_two_layers(negf, n, nsys):
    """A 2 x 2 block matrix: factors, then the inverse's blocks."""
    from libnegf_b200._lib import check, ptr_array
    import ctypes
    rng = np.random.default_rng(n)
    tol = 100 * 2.0 ** -53 * 2 * n + 1e-15
    mats = []
    for s in range(nsys):
        full = rng.standard_normal((2 * n, 2 * n)) + 1j * rng.standard_normal((2 * n, 2 * n)) + 6.0 * n * np.eye(2 * n)
        mats.append(full)
    blocks = [[negf.dzeros(n, n) for _ in range(4)] for _ in mats]
    for full, bl in zip(mats, blocks):
        for k, (i, j) in enumerate([(0, 0), (0, 1), (1, 0), (1, 1)]):
            bl[k].copy_(negf.to_device(full[i * n:(i + 1) * n, j * n:(j + 1) * n]))
    fill = (ctypes.c_uint8 * 4)()
    check(negf.load().negf_selected_inverse_batched(nsys, 2, n, ptr_array([b.data_ptr() for bl in blocks for b in bl]),
                                                    fill, 3, 0, 0, None))
    for full, bl in zip(mats, blocks):
        ref = np.linalg.inv(full)
        for k, (i, j) in enumerate([(0, 0), (0, 1), (1, 0), (1, 1)]):
            assert _rel(negf.to_host(bl[k]), ref[i * n:(i + 1) * n, j * n:(j + 1) * n]) <= tol


@pytest.mark.parametrize("n", [32, 33, 95, 128, 200, 300])
def test_triangular(negf, n):
    rng = np.random.default_rng(n)
    tol = 100 * 2.0 ** -53 * n
    P = _mat(rng, n)
    L, U = np.tril(P, -1) / (3.0 * n) + np.eye(n), np.triu(P)
    packed = np.tril(L, -1) + U
    B = rng.standard_normal((n, 7)) + 1j * rng.standard_normal((n, 7))
    dA = negf.to_device(packed)
    for side, ul, dg, ref in (("L", "U", "N", np.linalg.solve(U, B)), ("L", "L", "U", np.linalg.solve(L, B)),
                              ("R", "U", "N", np.linalg.solve(U.T, B).T), ("R", "L", "U", np.linalg.solve(L.T, B).T)):
        X = negf.to_device(B if side == "L" else B.T.copy())
        negf.be_trsm_(side, ul, "N", dg, 1.0, dA, X)
        assert _rel(negf.to_host(X), ref) <= tol
    negf.be_getri_(dA)
    assert _rel(negf.to_host(dA), np.linalg.inv(U) @ np.linalg.inv(L)) <= tol


def test_zero_pivot_named(negf):
    from libnegf_b200._lib import ptr_array, NEGF_ERR_SINGULAR
    import ctypes
    n = 70
    A = np.eye(n, dtype=complex)
    A[40, 40] = 0.0
    fill = (ctypes.c_uint8 * 1)()
    d = negf.to_device(A)
    rc = negf.load().negf_selected_inverse_batched(1, 1, n, ptr_array([d.data_ptr()]), fill, 1, 0, 0, None)
    assert rc == NEGF_ERR_SINGULAR and b"column 41" in negf.load().negf_last_error()
