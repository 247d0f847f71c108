"""Digit split of the mixed products at the ends of the exponent range (rows
scaled by one and by two powers of two), at the rows-per-CTA classes (k_pad 128,
256, 512, 1024) and for both storage orders of an operand.

Tolerance: 34 digit pairs are FP64-grade; the primitive's bar, 1e-12 relative to
|A||B|."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(rng, m, n):
    return rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))


@pytest.mark.parametrize("ops", ["NN", "CC", "TN"])
@pytest.mark.parametrize("k", [31, 128, 129, 256, 300, 513])
def test_exponent_range(negf, ops, k):
    rng = np.random.default_rng(k)
    m, n = 70, 45
    op = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
    A, B = _rand(rng, m, k), _rand(rng, k, n)
    # rows of op(A) and columns of op(B) across the range, products near one
    ea = rng.choice([-1005, -998, -990, -500, 0, 500, 970, 980], m)  # 2^980 2^20 sqrt(k): below overflow
    A2 = np.ldexp(A.real, ea[:, None]) + 1j * np.ldexp(A.imag, ea[:, None])
    for scale_b in (0, 20):
        B2 = B * 2.0 ** scale_b
        X, Y = op[ops[0]](A2), op[ops[1]](B2)
        if ops[0] == "C":
            X = A2.conj().T
        dC = negf.dzeros(m, n)
        negf.be_gemm_batched_(ops[0], ops[1], [(1.0, negf.to_device(X), negf.to_device(Y), 0.0, dC)], "mixed")
        got = negf.to_host(dC)
        # compare row by row with the scales taken out (exact powers of two)
        ref = (A @ B) * 2.0 ** scale_b
        g = np.ldexp(got.real, -ea[:, None]) + 1j * np.ldexp(got.imag, -ea[:, None])
        bound = 1e-12 * np.linalg.norm(A, axis=1)[:, None] * np.linalg.norm(B) * 2.0 ** scale_b
        ok = ea > -980  # below, the products themselves underflow partly
        assert np.all(np.abs(g - ref)[ok] <= bound[ok])
        low = ~ok
        # results near the denormal range: absolute rounding 2^-1074
        assert np.all(np.abs(g - ref)[low] <= bound[low] + np.ldexp(1.0, -1074 - ea[low])[:, None] * 4)
