"""What a user of the library has it do, as cases that can be timed and checked.

Three groups, over the sizes of the reference's tests and of the benchmark's
workloads (layers 4..1024, blocks 16..512, 1..64 energies):

* the drop-in layer: one call per block operation or per sweep of one system,
  as a program written against the reference's API makes them (latency, host
  work and launches count);
* the batched-energy solver: a resident plan of RGF + recursive Keldysh +
  transmission over many energies, FP64 or mixed precision, one device or an
  uneven batch of devices (throughput counts);
* whole one-shot calls: selected inverse of M(E), host-to-host solves.
"""

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "libnegf.jl_b200"))  # the package of the tree in use

ETA = 1e-2      # broadening of the one-call sweeps (DDRGF's closed interiors need it)
ETA_E = 1e-4    # broadening of the energy solver
MU_L, MU_R, KT = 0.1, -0.1, 0.025


def listed():
    return [
        # the smallest call: the inverses of a few blocks of the reference's test size
        dict(name="inv_24", kind="inv", count=4, n=24, ragged=0),
        # block products of one recursion step over many systems, odd sizes, B^H
        dict(name="gemm_137", kind="gemm", count=64, m=137, n=201, k=95, opA="N", opB="C", precision="fp64"),
        # one RGF of the reference's test shape (block sizes vary by +-4 as its generator's do)
        dict(name="rgf_10x32", kind="rgf", npl=10, b=32, spread=4),
        # one RGF of an ordinary device, one energy
        dict(name="rgf_16x256", kind="rgf", npl=16, b=256, spread=0),
        # one recursive Keldysh sweep with a full Hermitian tridiagonal Sigma^in, odd sizes
        dict(name="keldysh_20x100", kind="keldysh", npl=20, b=100, spread=4),
        # domain decomposition of a long thin device
        dict(name="ddrgf_1024x32", kind="ddrgf", npl=1024, b=32, spread=0),
        # energy solver on a small device with overlap matrix and Sigma(E)
        dict(name="solver_16x64_hs", kind="solver", devices="16x64", ne=64, precision="fp64", hs=True),
        # the benchmark's device, 64 of its energies, in both precision modes
        dict(name="solver_32x256_fp64", kind="solver", devices="32x256", ne=64, precision="fp64", hs=False),
        dict(name="solver_32x256_mixed", kind="solver", devices="32x256", ne=64, precision="mixed", hs=False),
        # uneven batch: devices of different layer counts and block sizes in one plan
        dict(name="batch_uneven_mixed", kind="solver", devices="8x384,21x190,30x256,64x128,96x64,50x33", ne=8,
             precision="mixed", hs=False),
        # block selected inverse of M(E) of wide layers, device outputs
        dict(name="selinv_16x512_mixed", kind="selinv", npl=16, b=512, ne=8, method=2, d1=0, precision="mixed"),
        # one-shot solve from a host program: plan, pass and host copies in every call
        dict(name="solve_24x128_host", kind="solve", npl=24, b=128, ne=24, precision="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["inv", "gemm", "rgf", "keldysh", "ddrgf", "solver", "solver", "solver", "selinv", "solve"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "inv":
        n = _log(rng, 8, 512)
        return dict(kind=kind, count=_log(rng, 1, max(2, min(256, 2 ** 22 // (n * n)))), n=n, ragged=rng.randint(0, n // 4))
    if kind == "gemm":
        m, n, k = (_log(rng, 16, 512) for _ in range(3))
        return dict(kind=kind, count=_log(rng, 1, 128), m=m, n=n, k=k, opA=rng.choice("NTC"), opB=rng.choice("NTC"),
                    precision=prec)
    if kind in ("rgf", "keldysh"):
        return dict(kind=kind, npl=_log(rng, 4, 64), b=_log(rng, 16, 400), spread=rng.choice([0, 4]))
    if kind == "ddrgf":
        return dict(kind=kind, npl=_log(rng, 100, 1000), b=_log(rng, 16, 64), spread=rng.choice([0, 4]))
    if kind == "solver":
        # work ~ layers x energies x b^3 stays below the largest listed case's
        room, devs, ne = 32 * 64 * 256 ** 3 // 2, [], _log(rng, 2, 32)
        for _ in range(rng.choice([1, 1, 2, 4])):
            b = _log(rng, 16, 384)
            n = max(3, min(_log(rng, 4, 96), room // (4 * ne * b ** 3)))
            devs.append("%dx%d" % (n, b))
        return dict(kind=kind, devices=",".join(devs), ne=ne, precision=prec, hs=len(devs) == 1 and rng.random() < 0.3)
    if kind == "selinv":
        method = rng.choice([0, 1, 2])
        b = _log(rng, 32, 400)
        n = 4 * _log(rng, 2, 8)  # four partitions of d1 interiors and a separator
        return dict(kind=kind, npl=n, b=b, ne=_log(rng, 1, 8), method=method, d1=n // 4 - 1 if method == 1 else 0,
                    precision=prec)
    return dict(kind="solve", npl=_log(rng, 4, 32), b=_log(rng, 16, 200), ne=_log(rng, 1, 24), precision=prec)


# --------------------------------------------------------------------------
# inputs, from the seed alone (host arrays)

def _cn(rng, shape, var):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * np.sqrt(var / 2.0)


def _sizes(c):
    s = c.get("spread", 0)
    return [c["b"] + ((5 * i) % (2 * s + 1) - s if s else 0) for i in range(c["npl"])]


def _sigma_parts(rng, n):
    B = _cn(rng, (n, n), 0.1 / n)
    Y = _cn(rng, (n, n), 1.0) / np.sqrt(n)
    return (B + B.conj().T) / 2.0, Y @ Y.conj().T + 0.1 * np.eye(n)


def _device(rng, sizes):
    """H blocks of unit spectral scale and the two lead self-energies."""
    Hd, Hu = [], []
    for b in sizes:
        A = _cn(rng, (b, b), 1.0) / np.sqrt(b)
        Hd.append((A + A.conj().T) / 2.0)
    for b, b2 in zip(sizes, sizes[1:]):
        Hu.append(_cn(rng, (b, b2), 0.25) / np.sqrt(b))
    XL, PL = _sigma_parts(rng, sizes[0])
    XR, PR = _sigma_parts(rng, sizes[-1])
    return dict(Hd=Hd, Hu=Hu, L=(XL, PL), R=(XR, PR), sL=XL - 0.05j * PL, sR=XR - 0.05j * PR)


def _sigma_E(parts, E):
    return (1.0 + 0.1 * E) * parts[0] - 0.05j * (1.0 + 0.5 * np.sin(2.0 * E)) * parts[1]


def _overlap(rng, sizes):
    Sd, Su = [], []
    for b in sizes:
        A = _cn(rng, (b, b), 1.0) / np.sqrt(b)
        Sd.append(np.eye(b) + 0.02 * (A + A.conj().T))
    for b, b2 in zip(sizes, sizes[1:]):
        Su.append(0.01 * _cn(rng, (b, b2), 1.0) / np.sqrt(b))
    return Sd, Su


def _M_blocks(d, z):
    """Block tridiagonal of M(E) = z I - H - Sigma."""
    n = len(d["Hd"])
    Md = [z * np.eye(h.shape[0]) - h for h in d["Hd"]]
    Md[0] = Md[0] - d["sL"]
    Md[n - 1] = Md[n - 1] - d["sR"]
    return Md, [-u for u in d["Hu"]], [-u.conj().T for u in d["Hu"]]


def _inputs(c, seed):
    rng = np.random.default_rng([20241, seed])
    k = c["kind"]
    if k == "inv":
        ns = [c["n"] - (7 * i) % (c["ragged"] + 1) for i in range(c["count"])]
        return [_cn(rng, (n, n), 1.0) / np.sqrt(n) + (0.3 + 0.1j) * np.eye(n) for n in ns]
    if k == "gemm":
        sa = (c["m"], c["k"]) if c["opA"] == "N" else (c["k"], c["m"])
        sb = (c["k"], c["n"]) if c["opB"] == "N" else (c["n"], c["k"])
        f = 1.0 / np.sqrt(c["k"])
        return [(_cn(rng, sa, 1.0) * f, _cn(rng, sb, 1.0)) for _ in range(c["count"])]
    if k in ("rgf", "keldysh", "ddrgf"):
        sizes = _sizes(c)
        d = _device(rng, sizes)
        Md, Mu, Ml = _M_blocks(d, rng.uniform(-1.0, 1.0) + 1j * ETA)
        Sd = Su = None
        if k == "keldysh":  # a scattering Sigma^in: Hermitian, diagonally dominant, coupled layers
            Sd = [_sigma_parts(rng, b)[1] for b in sizes]
            Su = [0.1 * _cn(rng, (b, b2), 1.0) / np.sqrt(b) for b, b2 in zip(sizes, sizes[1:])]
        return sizes, Md, Mu, Ml, Sd, Su
    if k == "solver":
        devs = []
        for text in c["devices"].split(","):
            n, b = (int(x) for x in text.split("x"))
            d = _device(rng, [b] * n)
            if c["hs"]:
                d["Sd"], d["Su"] = _overlap(rng, [b] * n)
            devs.append(d)
        E = np.concatenate([np.sort(rng.uniform(-1.0, 1.0, c["ne"])) for _ in devs])
        return devs, E
    d = _device(rng, [c["b"]] * c["npl"])
    return d, np.sort(rng.uniform(-1.0, 1.0, c["ne"]))


# --------------------------------------------------------------------------
# what a program has in hand before the call

class _View:
    """A library-owned device array for torch (no copy)."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _block_matrix(lib, sizes, Md, Mu, Ml, hermitian=False):
    bm = lib.BlockMatrix(sizes, None, {"in": 3, "out": 3}, False, hermitian)
    for i, a in enumerate(Md):
        bm.M[(i, i)] = lib.to_device(a)
    for i, a in enumerate(Mu):
        bm.M[(i, i + 1)] = lib.to_device(a)
    for i, a in enumerate(Ml or []):
        bm.M[(i + 1, i)] = lib.to_device(a)
    return bm


def _arena(shapes):
    """Column-major blocks of the given shapes in one zeroed allocation: (all of it, the blocks)."""
    flat = torch.zeros(sum(m * n for m, n in shapes), dtype=torch.complex128, device="cuda")
    blocks, o = [], 0
    for m, n in shapes:
        blocks.append(flat[o:o + m * n].view(n, m).t())
        o += m * n
    return flat, blocks


def _into_arena(bm, keys):
    """Give a BlockMatrix one allocation for all of its blocks (key order)."""
    flat, blocks = _arena([(bm.blockSizes[i], bm.blockSizes[j]) for i, j in keys])
    for k, b in zip(keys, blocks):
        bm.M[k] = b
    return flat


def _keys(n, lower=True):
    return sorted(p for i in range(n) for p in ((i, i), (i, i + 1), (i, i - 1))
                  if 0 <= p[1] < n and (lower or p[1] >= p[0]))


def prepare(c, seed):
    import libnegf_b200 as lib

    x = _inputs(c, seed)
    k = c["kind"]
    s = dict(case=c, lib=lib)
    if k == "inv":
        s["A"] = [lib.to_device(a) for a in x]
        s["flat"], s["out"] = _arena([a.shape for a in x])
    elif k == "gemm":
        s["flat"], out = _arena([(c["m"], c["n"])] * len(x))
        s["items"] = [(1.0, lib.to_device(a), lib.to_device(b), 0.0, cc) for (a, b), cc in zip(x, out)]
    elif k in ("rgf", "keldysh", "ddrgf"):
        sizes, Md, Mu, Ml, Sd, Su = x
        s["M"] = _block_matrix(lib, sizes, Md, Mu, Ml)
        if k == "rgf":
            s["out"] = lib.BlockMatrix(sizes, None, {"in": 3, "out": 3}, False, False)
            s["flat"] = _into_arena(s["out"], _keys(len(sizes)))
            s["aux"] = lib.allocate_aux_data_RGF(s["M"])
        elif k == "keldysh":
            s["S"] = _block_matrix(lib, sizes, Sd, Su, None, True)
            s["aux"] = lib.allocate_aux_data_Keldysh(s["M"], s["S"])
            s["flat"] = _into_arena(s["aux"].buffS, _keys(len(sizes), lower=False))
        else:
            s["aux"] = lib.allocate_aux_data_DDRGF(s["M"])
            s["flat"] = _into_arena(s["aux"][0].buffMout, _keys(len(sizes)))
    elif k == "solver":
        devs, E = x
        dev = [lib.Device(d["Hd"], d["Hu"], d["sL"], d["sR"]) for d in devs]
        kw = dict(eta=ETA_E, mu_l=MU_L, mu_r=MU_R, kT=KT, precision=c["precision"])
        if c["hs"]:
            dev[0].set_overlap(devs[0]["Sd"], devs[0]["Su"])
            kw["sigma_per_energy"] = True
        s["devices"] = dev
        s["stream"] = torch.cuda.Stream()  # a solver replays its pass as a CUDA graph on a stream of its own
        s["solver"] = lib.Solver(dev[0], c["ne"], **kw) if len(dev) == 1 else lib.BatchSolver(dev, [c["ne"]] * len(dev), **kw)
        if c["hs"]:
            s["solver"].set_self_energies([_sigma_E(devs[0]["L"], e) for e in E], [_sigma_E(devs[0]["R"], e) for e in E],
                                          s["stream"].cuda_stream)
        s["E"] = E
        n = c["ne"] * sum(sum(h.size for h in d["Hd"]) for d in devs)
        gr, gl, t = s["solver"].outputs()
        s["outs"] = (torch.as_tensor(_View(gr, n, "<c16"), device="cuda"), torch.as_tensor(_View(gl, n, "<c16"), device="cuda"),
                     torch.as_tensor(_View(t, 2 * len(E), "<f8"), device="cuda")[0::2])
    else:
        d, E = x
        s["device"] = lib.Device(d["Hd"], d["Hu"], d["sL"], d["sR"])
        s["E"] = E
        if k == "selinv":
            n, b, ne = c["npl"], c["b"], c["ne"]
            s["opts"] = lib.make_opts(eta=ETA, precision=c["precision"])
            s["outs"] = [torch.zeros(ne * m * b * b, dtype=torch.complex128, device="cuda") for m in (n, n - 1, n - 1)]
    return s


def run(s):
    lib, c = s["lib"], s["case"]
    k = c["kind"]
    if k == "inv":
        lib.be_inv_batched_(s["A"], s["out"])
        return s["flat"]
    if k == "gemm":
        lib.be_gemm_batched_(c["opA"], c["opB"], s["items"], c["precision"])
        return s["flat"]
    if k == "rgf":
        lib.bndiag_of_inv_rgf_local_(s["out"], s["M"], s["aux"])
        return s["flat"]
    if k == "keldysh":
        lib.keldyshndiag_(s["M"], s["S"], s["aux"])
        return s["flat"]
    if k == "ddrgf":
        lib.bndiag_of_inv_ddrgf_(s["M"], s["aux"])
        return s["flat"]
    if k == "solver":
        st = s["stream"].cuda_stream
        s["solver"].set_energies(s["E"], st)
        s["solver"].run(st)
        return list(s["outs"])
    if k == "selinv":
        E = s["E"]
        lib._lib.check(lib.load().negf_device_selected_inverse(
            s["device"].handle, len(E), E.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.byref(s["opts"]),
            c["method"], 1 if c["d1"] else 0, lib._lib.int_array([c["d1"]]) if c["d1"] else None,
            s["outs"][0].data_ptr(), s["outs"][1].data_ptr(), s["outs"][2].data_ptr(), 1, lib.stream_handle()))
        return list(s["outs"])
    gr, gl, t = s["device"].solve(s["E"], eta=ETA_E, mu_l=MU_L, mu_r=MU_R, kT=KT, precision=c["precision"])
    return [gr[0][0].base, gl[0][0].base, t]  # the whole arrays that the blocks are views of


# --------------------------------------------------------------------------
# what one pass cannot do without: every input read and every output written
# once; per layer one inversion (8 b^3) and the products (8 b^3 each) of the
# recursion that gives the wanted blocks

def work(c):
    k, z = c["kind"], 16.0
    if k == "inv":
        ns = [c["n"] - (7 * i) % (c["ragged"] + 1) for i in range(c["count"])]
        return dict(bytes=2 * z * sum(n * n for n in ns), flops=8.0 * sum(n ** 3 for n in ns))
    if k == "gemm":
        m, n, kk = c["m"], c["n"], c["k"]
        return dict(bytes=c["count"] * z * (m * kk + kk * n + m * n), flops=c["count"] * 8.0 * m * n * kk)
    if k in ("rgf", "ddrgf", "keldysh"):
        sizes = _sizes(c)
        d, u = sum(b * b for b in sizes), sum(a * b for a, b in zip(sizes, sizes[1:]))
        cube = sum(b ** 3 for b in sizes)
        if k == "keldysh":
            return dict(bytes=z * (3 * d + 4 * u), flops=8.0 * cube * (1 + 3 + 10))
        return dict(bytes=z * (2 * d + 4 * u), flops=8.0 * cube * (1 + 3 + 3))
    if k == "solver":
        by = fl = 0.0
        for text in c["devices"].split(","):
            n, b = (int(x) for x in text.split("x"))
            by += z * b * b * (2 * n + 1) + c["ne"] * z * 2 * n * b * b
            fl += c["ne"] * 8.0 * n * b ** 3 * (1 + 12)
        return dict(bytes=by, flops=fl)
    n, b, ne = c["npl"], c["b"], c["ne"]
    if k == "selinv":
        return dict(bytes=z * b * b * (2 * n + 1 + ne * (3 * n - 2)), flops=ne * 8.0 * n * b ** 3 * (1 + 3 + 3))
    return dict(bytes=z * b * b * (2 * n + 1 + ne * 2 * n), flops=ne * 8.0 * n * b ** 3 * (1 + 12))


# --------------------------------------------------------------------------
# the same outputs from plain torch in 64 bits

def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda" if torch.cuda.is_available() else "cpu")


def _tri_inverse(Md, Mu, Ml):
    """Block tridiagonal of M^{-1}, batched: block LU from the last layer up, then down."""
    n = len(Md)
    g, R, L = [None] * n, [None] * n, [None] * n
    g[n - 1] = torch.linalg.inv(Md[n - 1])
    for i in range(n - 2, -1, -1):
        R[i] = Mu[i] @ g[i + 1]
        L[i] = g[i + 1] @ Ml[i]
        g[i] = torch.linalg.inv(Md[i] - Mu[i] @ L[i])
    d, u, l = [g[0]], [], []
    for i in range(n - 1):
        u.append(-d[i] @ R[i])
        l.append(-L[i] @ d[i])
        d.append(g[i + 1] - L[i] @ u[i])
    return d, u, l, g, R, L


def _h(a):
    return a.mH


def _exact_solver(d, E, hs):
    n, ne = len(d["Hd"]), len(E)
    zE = _t(E + 1j * ETA_E).view(ne, 1, 1)
    sL = _t(np.stack([_sigma_E(d["L"], e) if hs else d["sL"] for e in E]))
    sR = _t(np.stack([_sigma_E(d["R"], e) if hs else d["sR"] for e in E]))
    Md = [zE * _t(d["Sd"][i] if hs else np.eye(h.shape[0]).astype(complex)) - _t(h) for i, h in enumerate(d["Hd"])]
    Md[0] = Md[0] - sL
    Md[n - 1] = Md[n - 1] - sR
    Mu = [(zE * _t(d["Su"][i]) if hs else 0.0) - _t(u) for i, u in enumerate(d["Hu"])]
    Ml = [(zE * _h(_t(d["Su"][i])) if hs else 0.0) - _h(_t(u)) for i, u in enumerate(d["Hu"])]
    dd, u, _, g, R, L = _tri_inverse(Md, Mu, Ml)
    del u
    # G^R_{i,0} down from the first layer; G^R_{i,N-1} from the right-connected
    # last column F_i = -g_i M_{i,i+1} F_{i+1}
    F = [None] * n
    F[n - 1] = g[n - 1]
    for i in range(n - 2, -1, -1):
        F[i] = -g[i] @ (Mu[i] @ F[i + 1])
    gamL, gamR = 1j * (sL - _h(sL)), 1j * (sR - _h(sR))
    fL = _t(1.0 / (1.0 + np.exp((E - MU_L) / KT))).view(ne, 1, 1)
    fR = _t(1.0 / (1.0 + np.exp((E - MU_R) / KT))).view(ne, 1, 1)
    C0, CN, gl = dd[0], F[0], []
    T = torch.einsum("eij,eji->e", gamL @ CN, gamR @ _h(CN)).real
    for i in range(n):
        if i:
            C0 = -L[i - 1] @ C0
            CN = F[i] - L[i - 1] @ CN
        gl.append(1j * (fL * (C0 @ gamL @ _h(C0)) + fR * (CN @ gamR @ _h(CN))))
    return dd, gl, T


def _colmajor(blocks):
    """nE x N x b x b column-major block order, flat (energy, layer, column, row)."""
    return torch.stack([x.mT for x in blocks], 1).reshape(-1)


def _flat(blocks):
    """The blocks one after the other, column-major."""
    return torch.cat([torch.as_tensor(b).mT.reshape(-1) for b in blocks])


def exact(c, seed):
    x = _inputs(c, seed)
    k = c["kind"]
    if k == "inv":
        return _flat([np.linalg.inv(a) for a in x])
    if k == "gemm":
        f = dict(N=lambda a: a, T=lambda a: a.T, C=lambda a: a.conj().T)
        return _flat([f[c["opA"]](a) @ f[c["opB"]](b) for a, b in x])
    if k in ("rgf", "ddrgf", "keldysh"):
        sizes, Md, Mu, Ml, Sd, Su = x
        n = len(sizes)
        Md, Mu, Ml = ([_t(a) for a in v] for v in (Md, Mu, Ml))
        d, u, l, g, R, L = _tri_inverse(Md, Mu, Ml)
        if k != "keldysh":
            got = {(i, i): d[i] for i in range(n)}
            got.update({(i, i + 1): u[i] for i in range(n - 1)})
            got.update({(i + 1, i): l[i] for i in range(n - 1)})
            return _flat([got[p] for p in _keys(n)])
        # G S G^H: up with the right-connected operator, down with G
        Sd, Su = [_t(a) for a in Sd], [_t(a) for a in Su]
        A, B = [a.clone() for a in Sd], [a.clone() for a in Su]
        for i in range(n - 2, -1, -1):
            A[i] = A[i] - R[i] @ _h(B[i])
            B[i] = B[i] - R[i] @ A[i + 1]
            A[i] = A[i] - B[i] @ _h(R[i])
        G = [g[i] @ A[i] @ _h(g[i]) for i in range(n)]
        U = [d[i] @ B[i] @ _h(g[i + 1]) for i in range(n - 1)]
        for i in range(n - 1):
            G[i + 1] = G[i + 1] - _h(U[i]) @ _h(L[i])
            U[i] = U[i] - G[i] @ _h(L[i])
            G[i + 1] = G[i + 1] - L[i] @ U[i]
        got = {(i, i): G[i] for i in range(n)}
        got.update({(i, i + 1): U[i] for i in range(n - 1)})
        return _flat([got[p] for p in _keys(n, lower=False)])
    if k == "solver":
        devs, E = x
        gr, gl, t = [], [], []
        for q, d in enumerate(devs):
            a, b, T = _exact_solver(d, E[q * c["ne"]:(q + 1) * c["ne"]], c["hs"])
            gr.append(_colmajor(a))
            gl.append(_colmajor(b))
            t.append(T)
        return [torch.cat(v) for v in (gr, gl, t)]
    d, E = x
    if k == "selinv":
        M = [_M_blocks(d, e + 1j * ETA) for e in E]
        Md, Mu, Ml = ([_t(np.stack([m[j][i] for m in M])) for i in range(len(M[0][j]))] for j in range(3))
        dd, u, l = _tri_inverse(Md, Mu, Ml)[:3]
        return [_colmajor(v) for v in (dd, u, l)]
    dd, gl, T = _exact_solver(d, E, False)
    return [_colmajor(dd), _colmajor(gl), T]
