"""FP64 products at the edges of the 3M kernels' tiles: 16 x 16 tiles (few
problems) and 32 x 32 tiles (many), every op pair, remainders in m, n and k, a
missing product (k = 0) and padded leading dimensions.

Tolerance: the three real products of length k and their combination round to
at most (k + 8) u (|Ar| + |Ai|)(|Br| + |Bi|) per element and product; in the
Frobenius norm 6 (k + 8) u |A| |B|, and 4 u |C| for the beta term."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPS = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
SHAPES = [(1, 1, 1), (16, 16, 16), (17, 15, 31), (32, 32, 33), (33, 47, 64), (5, 64, 1), (100, 3, 48), (31, 96, 17)]


def _rand(rng, m, n):
    return rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))


def _dev(negf, x):
    d = negf.dzeros(*x.shape)  # column-major also where a dimension is 1
    d.copy_(negf.to_device(x))
    return d


@pytest.mark.parametrize("ops", [a + b for a in "NTC" for b in "NTC"])
@pytest.mark.parametrize("copies", [1, 24])  # 24 copies of the shapes: more than 96 tiles of 32 x 32
def test_tiles(negf, ops, copies):
    rng = np.random.default_rng(7)
    tA, tB = ops
    alpha, beta = 0.8 - 0.3j, -0.4 + 1.1j
    items, refs = [], []
    for c in range(copies):
        for m, n, k in SHAPES:
            A = _rand(rng, *((m, k) if tA == "N" else (k, m)))
            B = _rand(rng, *((k, n) if tB == "N" else (n, k)))
            C = _rand(rng, m, n)
            big = negf.dzeros(m + 3, n)  # leading dimension m + 3
            big[:m, :].copy_(negf.to_device(C))
            items.append((alpha, _dev(negf, A), _dev(negf, B), beta, big[:m, :]))
            refs.append((alpha * OPS[tA](A) @ OPS[tB](B) + beta * C, k, np.linalg.norm(A) * np.linalg.norm(B),
                         np.linalg.norm(C)))
    negf.be_gemm_batched_(tA, tB, items)
    for it, (ref, k, ab, c) in zip(items, refs):
        err = np.linalg.norm(negf.to_host(it[4]) - ref)
        assert err <= 2.0 ** -53 * (6 * (k + 8) * ab + 4 * c)


@pytest.mark.parametrize("count", [2, 200])
def test_no_product(negf, count):
    """k = 0: C = beta Cin + diag I."""
    from libnegf_b200 import _lib
    rng = np.random.default_rng(3)
    n = 37
    cin = [_rand(rng, n, n) for _ in range(count)]
    dC = [negf.to_device(c) for c in cin]
    out = [negf.dzeros(n, n) for _ in range(count)]
    arr = (_lib.ZGemmProblem * count)()
    for p, a, o in zip(arr, dC, out):
        p.Cin, p.C, p.m, p.n, p.k = a.data_ptr(), o.data_ptr(), n, n, 0
        p.lda = p.ldb = 1
        p.ldc = p.ldcin = n
        p.beta[0], p.diag[0], p.diag[1] = 2.0, 0.5, -1.0
    assert negf.load().negf_zgemm_batched(b"N", b"N", count, arr, ctypes.c_void_p(None)) == 0
    for c, o in zip(cin, out):
        assert np.array_equal(negf.to_host(o), 2.0 * c + (0.5 - 1.0j) * np.eye(n))
