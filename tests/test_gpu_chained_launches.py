"""One-shot sweeps whose launches overlap their predecessors' ends: block sizes
that keep every pair of launches on one side of the line (CTAs of both against
the SMs of the GPU) and sizes where it alternates, called often, so that a
missing wait would show as a run that differs from the first.

Tolerance: two backward-stable inversions differ by no more than n u cond, with
n the order of the whole matrix and u = 2^-53."""

import numpy as np
import pytest

from conftest import rel_fro
from oracle.blockmatrix import band_of_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npl,b", [(24, 5), (12, 32), (8, 40), (8, 112), (6, 144), (4, 272), (1, 64)])
def test_rgf_repeats(negf, npl, b):
    rng = np.random.default_rng(npl * b)
    sizes = [b + (i % 3) - 1 for i in range(npl)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = off[-1]
    D = np.zeros((n, n), complex)
    M = negf.BlockMatrix(sizes)
    for i in range(npl):
        for j in range(max(0, i - 1), min(npl, i + 2)):
            a = (rng.standard_normal((sizes[i], sizes[j])) + 1j * rng.standard_normal((sizes[i], sizes[j]))) / np.sqrt(b)
            if i == j:
                a += 4.0 * np.eye(sizes[i])
            D[off[i]:off[i + 1], off[j]:off[j + 1]] = a
            M.M[(i, j)] = negf.to_device(a)
    ref = band_of_dense(np.linalg.inv(D), sizes, {"in": 3, "out": 3})
    first = None
    for _ in range(12):
        out = negf.BlockMatrix(sizes)
        negf.bndiag_of_inv_rgf_local_(out, M)
        G = negf.bm_to_dense(out)
        if first is None:
            first = G
            assert rel_fro(G, ref) <= 2.0 ** -53 * n * np.linalg.cond(D)
        assert np.array_equal(G, first)
