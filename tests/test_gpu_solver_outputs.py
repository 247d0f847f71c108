"""Every choice of outputs of the energy solver (G^R, G^<, T), on devices of one,
two, three and seven layers, against the dense inverse: with all three in one
pass, without G^R (its blocks live in a ring), without the transmission chain, and
without G^< (plain RGF, no blocks below the diagonal).

Tolerance: G by two backward-stable inversions, n u cond(M) |G| each (n the order
of M, u = 2^-53); G^< and T are products of two and four factors of that kind.
Mixed products round to 1.5e-15 of |A||B|, 14 u: 16 times the bound."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ETA, MU_L, MU_R, KT = 1e-2, 0.1, -0.1, 0.025
DEVICES = [[20], [17, 17], [24, 9, 24], [16, 5, 40, 33, 8, 21, 16], [120, 130, 120]]
E = np.array([-0.4, 0.05, 0.3])


def _cn(rng, m, n):
    return (rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))) / np.sqrt(m + n)


def _system(sizes):
    rng = np.random.default_rng(sum(sizes))
    Hd = [(a + a.conj().T) / 2 for a in (_cn(rng, b, b) for b in sizes)]
    Hu = [0.5 * _cn(rng, a, b) for a, b in zip(sizes, sizes[1:])]
    sig = []
    for b in (sizes[0], sizes[-1]):
        y = _cn(rng, b, b)
        sig.append(0.1 * (y + y.conj().T) - 0.1j * (y @ y.conj().T + 0.1 * np.eye(b)))
    return Hd, Hu, sig


def _dense(sizes, Hd, Hu, sig, e):
    o = np.concatenate([[0], np.cumsum(sizes)])
    s = [slice(o[i], o[i + 1]) for i in range(len(sizes))]
    M = (e + 1j * ETA) * np.eye(o[-1], dtype=complex)
    for i, h in enumerate(Hd):
        M[s[i], s[i]] -= h
    for i, u in enumerate(Hu):
        M[s[i], s[i + 1]] = -u
        M[s[i + 1], s[i]] = -u.conj().T
    M[s[0], s[0]] -= sig[0]
    M[s[-1], s[-1]] -= sig[1]
    G = np.linalg.inv(M)
    gam = [1j * (x - x.conj().T) for x in sig]
    f = [1.0 / (1.0 + np.exp((e - mu) / KT)) for mu in (MU_L, MU_R)]
    less = 1j * (f[0] * G[:, s[0]] @ gam[0] @ G[:, s[0]].conj().T + f[1] * G[:, s[-1]] @ gam[1] @ G[:, s[-1]].conj().T)
    t = np.trace(gam[0] @ G[s[0], s[-1]] @ gam[1] @ G[s[0], s[-1]].conj().T).real
    err, g, q = 2.0 ** -53 * o[-1] * np.linalg.cond(M), np.linalg.norm(G), max(np.linalg.norm(x) for x in gam)
    return [G[x, x] for x in s], [less[x, x] for x in s], t, 2 * err * g, 8 * err * g * g * q, 8 * err * (g * q) ** 2


@pytest.fixture(scope="module")
def systems():
    sys_ = [_system(s) for s in DEVICES]
    return sys_, [[_dense(s, *x, e) for e in E] for s, x in zip(DEVICES, sys_)]


def _check(got, ref, want, k):
    gr, gl, t = got
    assert [x is not None for x in got] == list(want)
    for e, (dr, dl, dt, tr, tl, tt) in enumerate(ref):
        for i in range(len(dr)):
            assert gr is None or np.linalg.norm(gr[e][i] - dr[i]) <= k * tr
            assert gl is None or np.linalg.norm(gl[e][i] - dl[i]) <= k * tl
        assert t is None or abs(t[e] - dt) <= k * tt


WANT = [(r, l, t) for r in (0, 1) for l in (0, 1) for t in (0, 1) if r or l or t]


@pytest.mark.parametrize("precision,k", [("fp64", 1), ("mixed", 16)])
@pytest.mark.parametrize("want", WANT)
def test_outputs(negf, systems, want, precision, k):
    import torch
    sys_, refs = systems
    kw = dict(eta=ETA, mu_l=MU_L, mu_r=MU_R, kT=KT, want_gr=want[0], want_gl=want[1], want_t=want[2], precision=precision)
    devs = [negf.Device(Hd, Hu, *sig) for Hd, Hu, sig in sys_]
    for d, ref in zip(devs, refs):  # one call each: direct launches, downloads by layer
        _check(d.solve(E, **kw), ref, want, k)
    batch = negf.BatchSolver(devs, [len(E)] * len(devs), **kw)
    stream = torch.cuda.Stream()
    for _ in range(3):  # captured, then replayed
        batch.set_energies(np.tile(E, len(devs)), stream.cuda_stream)
        batch.run(stream.cuda_stream)
    stream.synchronize()
    batch.check()
    gr, gl, t = batch.host_outputs()
    for i, ref in enumerate(refs):
        _check([x and x[i] if x is not None else None for x in (gr, gl)] + [t[i] if t is not None else None], ref, want, k)
