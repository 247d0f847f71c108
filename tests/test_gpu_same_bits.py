"""The energy solver's results of one energy are the same to the last bit whatever
the number of energies beside it, as long as the block sizes are the same."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cn(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("b", [24, 70, 130])
def test_energies(negf, precision, b):
    """One energy alone, among others, and among those of a second device of the
    same block size."""
    rng = np.random.default_rng(b)
    devs = []
    for npl in (5, 3):
        Hd = [(a + a.conj().T) / 2 for a in (_cn(rng, b, b) / np.sqrt(2 * b) for _ in range(npl))]
        Hu = [0.3 * _cn(rng, b, b) / np.sqrt(b) for _ in range(npl - 1)]
        s = -0.05j * np.eye(b)
        devs.append(negf.Device(Hd, Hu, s, s))
    E = np.linspace(-0.8, 0.9, 40)
    alone = devs[0].solve(E[7:8], eta=1e-3, precision=precision)
    many = devs[0].solve(E, eta=1e-3, precision=precision)
    both = negf.BatchSolver(devs, [40, 40], eta=1e-3, precision=precision)
    both.set_energies(np.concatenate([E, E]))
    both.run()
    gr, gl, t = both.host_outputs()
    for x, y, z in ((alone[0], many[0], gr[0]), (alone[1], many[1], gl[0])):
        for i in range(5):
            assert np.array_equal(x[0][i], y[7][i]) and np.array_equal(x[0][i], z[7][i])
    assert alone[2][0] == many[2][7] == t[0][7]
