"""One-shot calls whose launches overlap their predecessors' ends, beyond RGF: the
Keldysh sweep, DDRGF, the unpivoted selected inverse (LU diagonal blocks and
solves, triangular joins) and mixed products (digit split, INT8 kernel), at sizes
on both sides of the line (CTAs of two launches against the SMs of the GPU),
called often, so that a missing wait would show as a run that differs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPEATS = 12


def _cn(rng, m, n):
    return (rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))) / np.sqrt(m + n)


def _dev(rng, npl, b):
    import libnegf_b200 as negf
    Hd = [(a + a.conj().T) / 2 for a in (_cn(rng, b, b) for _ in range(npl))]
    Hu = [0.5 * _cn(rng, b, b) for _ in range(npl - 1)]
    s = -0.05j * np.eye(b)
    M = np.zeros((npl * b, npl * b), complex)
    for i in range(npl):
        M[i * b:(i + 1) * b, i * b:(i + 1) * b] = (0.1 + 5e-2j) * np.eye(b) - Hd[i] - (s if i in (0, npl - 1) else 0)
        if i + 1 < npl:
            M[i * b:(i + 1) * b, (i + 1) * b:(i + 2) * b] = -Hu[i]
            M[(i + 1) * b:(i + 2) * b, i * b:(i + 1) * b] = -Hu[i].conj().T
    return negf.Device(Hd, Hu, s, s), M


@pytest.mark.parametrize("npl,b", [(1, 30), (2, 33), (12, 5), (8, 40), (4, 112), (4, 144), (3, 272)])
def test_keldysh(negf, npl, b):
    """G S G^H on the block tridiagonal; bound: n u cond(M) for each factor G."""
    rng = np.random.default_rng(npl * b)
    _, D = _dev(rng, npl, b)
    n = npl * b
    sl = [slice(i * b, (i + 1) * b) for i in range(npl)]
    S = np.zeros((n, n), complex)
    for i in range(npl):
        y = _cn(rng, b, b)
        S[sl[i], sl[i]] = y @ y.conj().T + np.eye(b)
        if i + 1 < npl:
            S[sl[i], sl[i + 1]] = 0.1 * _cn(rng, b, b)
            S[sl[i + 1], sl[i]] = S[sl[i], sl[i + 1]].conj().T
    G = np.linalg.inv(D)
    ref = G @ S @ G.conj().T
    bound = 8 * 2.0 ** -53 * n * np.linalg.cond(D) * np.linalg.norm(G) ** 2 * np.linalg.norm(S, 2)
    M = negf.BlockMatrix([b] * npl)
    T = negf.BlockMatrix([b] * npl, None, {"in": 3, "out": 3}, False, True)
    for i in range(npl):
        for j in range(max(0, i - 1), min(npl, i + 2)):
            M.M[(i, j)] = negf.to_device(D[sl[i], sl[j]])
            if j >= i:
                T.M[(i, j)] = negf.to_device(S[sl[i], sl[j]])
    first = None
    for _ in range(REPEATS):
        aux = negf.allocate_aux_data_Keldysh(M, T)
        negf.keldyshndiag_(M, T, aux)
        got = {k: negf.to_host(v) for k, v in aux.buffS.M.items() if k[1] >= k[0]}
        if first is None:
            first = got
            for (i, j), v in got.items():
                assert np.linalg.norm(v - ref[sl[i], sl[j]]) <= bound
        assert all(np.array_equal(v, first[k]) for k, v in got.items())


@pytest.mark.parametrize("precision,k", [("fp64", 1), ("mixed", 16)])
@pytest.mark.parametrize("method,levels", [("selinv", None), ("ddrgf", [2]), ("rgf", None)])
@pytest.mark.parametrize("npl,b", [(6, 24), (6, 65), (4, 130)])
def test_selected_inverse(negf, npl, b, method, levels, precision, k):
    """Bound: n u cond(M) |G|, twice that of a block (no pivoting across blocks in
    either method; eta = 5e-2 keeps the interior domains well conditioned)."""
    rng = np.random.default_rng(npl * b)
    dev, M = _dev(rng, npl, b)
    if method == "ddrgf" and npl == 4:
        levels = [1]
    G = np.linalg.inv(M)
    bound = 2 * k * 2.0 ** -53 * npl * b * np.linalg.cond(M) * np.linalg.norm(G)
    first = None
    for _ in range(REPEATS):
        r = dev.selected_inverse([0.1], method, precision, eta=5e-2, levels=levels)
        got = [x for part in r for x in part[0]]
        if first is None:
            first = [x.copy() for x in got]
            for i in range(npl):
                assert np.linalg.norm(r[0][0][i] - G[i * b:(i + 1) * b, i * b:(i + 1) * b]) <= bound
        assert all(np.array_equal(x, y) for x, y in zip(got, first))


@pytest.mark.parametrize("n", [20, 130, 300])
def test_mixed_products(negf, n):
    """Bar of the mixed primitive: 1e-12 of |A||B|."""
    rng = np.random.default_rng(n)
    A, B = _cn(rng, n, n), _cn(rng, n, n)
    dA, dB = negf.to_device(A), negf.to_device(B)
    first = None
    for _ in range(REPEATS):
        o = negf.dzeros(n, n)
        negf.be_gemm_batched_("N", "C", [(1.0, dA, dB, 0.0, o)], "mixed")
        got = negf.to_host(o)
        if first is None:
            first = got
            assert np.linalg.norm(got - A @ B.conj().T) <= 1e-12 * np.linalg.norm(A) * np.linalg.norm(B)
        assert np.array_equal(got, first)
