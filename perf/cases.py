"""Timed cases of the framework's public entry points.

Each case is one call as a user's program makes it: H applied to a block of
vectors in either precision, the inner products of a projection, and whole
eigensolves.  Vectors live on the GPU; the handle (operator tables, workspace)
is made once and kept, as a program that iterates keeps it.

The operator is the reference's two-electron sinc-DVR Hamiltonian on NN = 2N+1
points per axis (D = NN^6 elements per vector, spacing 2 bohr), as the tests
and the benchmark build it."""
import ctypes
import math

import numpy as np
import torch

import doublyexcited_b200 as de
from doublyexcited_b200._lib import de_complex, de_gmres, de_stats

DELTA, CHARGE = 2.0, 2.0
THETAS = [0.20, 0.25, 0.30, 0.35, 0.40, 0.45, 0.50]


def listed():
    return [
        # H on one complex128 vector at the smallest grid of the serving mix:
        # a call whose cost is launches and latency
        {"name": "matvec_c128_n3_v1", "kind": "matvec", "storage": "c128", "n": 3, "nvec": 1, "theta": 0.3},
        # the block matvec of a four-resonance solve in the serving mix
        {"name": "matvec_c128_n4_v4", "kind": "matvec", "storage": "c128", "n": 4, "nvec": 4, "theta": 0.3},
        # the reference's logged configuration, one column: every outer step of
        # the one-resonance solve, and every product of the plain form
        {"name": "matvec_c128_n6_v1", "kind": "matvec", "storage": "c128", "n": 6, "nvec": 1, "theta": 0.2},
        # the outer products of the eight-resonance solve
        {"name": "matvec_c128_n8_v8", "kind": "matvec", "storage": "c128", "n": 8, "nvec": 8, "theta": 0.35},
        # the block-matvec throughput configuration: 16 vectors of 753 MB
        {"name": "matvec_c128_n9_v16", "kind": "matvec", "storage": "c128", "n": 9, "nvec": 16, "theta": 0.35},
        # the largest grid that the tests run, one vector of 1.4 GB
        {"name": "matvec_c128_n10_v1", "kind": "matvec", "storage": "c128", "n": 10, "nvec": 1, "theta": 0.35},
        # the mixed form's inner-solve products: one column at the two logged
        # grids, and the block of the eight-resonance solve
        {"name": "matvec_c64_n5_v1", "kind": "matvec", "storage": "c64", "n": 5, "nvec": 1, "theta": 0.2},
        {"name": "matvec_c64_n6_v1", "kind": "matvec", "storage": "c64", "n": 6, "nvec": 1, "theta": 0.2},
        {"name": "matvec_c64_n8_v8", "kind": "matvec", "storage": "c64", "n": 8, "nvec": 8, "theta": 0.35},
        # the inner products of a harmonic projection: 8 basis vectors against 16
        {"name": "dots_n6_8x16", "kind": "dots", "n": 6, "nbra": 8, "nket": 16, "hermitian": True},
        # the plain form's block solve: the first two outer iterations of a
        # four-resonance run (preconditioner, orthogonalisation, projection)
        {"name": "solve_fp64_n5_nev4", "kind": "solve", "precision": "fp64", "n": 5, "nev": 4, "theta": 0.3,
         "sigma": -0.78, "ns": 5, "maxit": 2, "tol": 1e-14},
        # the benchmark's workload: one resonance in the mixed form, from a
        # seeded start to convergence
        {"name": "solve_mixed_n6", "kind": "solve", "precision": "mixed", "n": 6, "nev": 1, "theta": 0.2,
         "sigma": -0.7131541429, "ns": 5, "maxit": 200, "tol": 1e-9},
    ]


def draw(rng):
    kind = rng.choice(["c128", "c128", "c128", "c64", "c64", "c64", "dots", "dots", "fp64", "mixed"])
    if kind in ("c128", "c64"):
        n = rng.randint(2, 10)
        most = min(16, 12_000_000_000 // (16 * (2 * n + 1) ** 6))  # the largest listed block
        nvec = max(1, min(most, int(round(math.exp(rng.uniform(0.0, math.log(most + 0.5)))))))
        return {"kind": "matvec", "storage": kind, "n": n, "nvec": nvec, "theta": rng.choice(THETAS)}
    if kind == "dots":
        n = rng.randint(3, 6)
        nbra, nket = (max(1, int(round(math.exp(rng.uniform(0.0, math.log(24.0)))))) for _ in range(2))
        return {"kind": "dots", "n": n, "nbra": nbra, "nket": nket, "hermitian": rng.random() < 0.7}
    if kind == "fp64":
        return {"kind": "solve", "precision": "fp64", "n": rng.randint(3, 5), "nev": rng.randint(1, 4),
                "theta": rng.choice(THETAS), "sigma": -round(rng.uniform(0.70, 0.80), 3), "ns": rng.randint(3, 5),
                "maxit": rng.randint(1, 2), "tol": 1e-14}
    return {"kind": "solve", "precision": "mixed", "n": rng.randint(4, 6), "nev": 1, "theta": 0.2,
            "sigma": -round(rng.uniform(0.711, 0.716), 5), "ns": rng.randint(4, 5), "maxit": 200, "tol": 1e-9}


def _dim(case):
    return (2 * case["n"] + 1) ** 6


def _vectors(rows, dim, seed, dtype=torch.complex128):
    """Complex-Gaussian vectors of unit mean square, one to a row."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000003) + 17)
    return torch.randn(rows, dim, dtype=dtype, device="cuda", generator=g)


def _on_torch_stream(problem):
    problem.set_stream(torch.cuda.current_stream().cuda_stream)
    return problem


def prepare(case, seed):
    dim = _dim(case)
    if case["kind"] == "matvec":
        mixed = case["storage"] == "c64"
        x = _vectors(case["nvec"], dim, seed, torch.complex64 if mixed else torch.complex128)
        p = _on_torch_stream(de.Problem(n=case["n"], delta=DELTA, theta=case["theta"], charge=CHARGE,
                                        precision="mixed" if mixed else "fp64"))
        return {"case": case, "problem": p, "x": x, "y": torch.empty_like(x)}
    if case["kind"] == "dots":
        p = _on_torch_stream(de.Problem(n=case["n"], delta=DELTA, theta=0.2, charge=CHARGE))
        both = _vectors(case["nbra"] + case["nket"], dim, seed) / math.sqrt(dim)
        return {"case": case, "problem": p, "bras": both[:case["nbra"]], "kets": both[case["nbra"]:],
                "out": np.empty((case["nket"], case["nbra"]), np.complex128)}
    p = _on_torch_stream(de.Problem(n=case["n"], delta=DELTA, theta=case["theta"], charge=CHARGE,
                                    precision=case["precision"]))
    # singlet starts: symmetric under electron exchange, unit norm
    x = _vectors(case["nev"], dim, seed).view(case["nev"], p.m, p.m)
    x = (x + x.transpose(1, 2)).reshape(case["nev"], dim)
    x = x / torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return {"case": case, "problem": p, "start": x, "x": torch.empty_like(x),
            "e": np.empty(case["nev"], np.complex128)}


def _check(status, where):
    if status != de.DE_OK:
        raise de.DeError(status, where, (de.lib().de_last_error() or b"").decode())


def run(state):
    case, p = state["case"], state["problem"]
    if case["kind"] == "matvec":
        call = p.matblock32_d if case["storage"] == "c64" else p.matblock_d
        call(state["x"].data_ptr(), state["y"].data_ptr(), case["nvec"])
        return state["y"]
    if case["kind"] == "dots":
        out = state["out"]
        _check(de.lib().de_dots_d(p.handle, state["bras"].data_ptr(), state["kets"].data_ptr(), p.dim, case["nbra"],
                                  case["nket"], out.ctypes.data, int(case["hermitian"])), "de_dots_d")
        return out
    x, e = state["x"], state["e"]
    x.copy_(state["start"])
    gm, st = de_gmres(5, 1, 1e-3, 0), de_stats()
    _check(de.lib().de_gplmr_eig_d(p.handle, x.data_ptr(), e.ctypes.data, p.m, p.m, de_complex(case["sigma"], 0.0),
                                   case["nev"], case["ns"], case["maxit"], case["tol"], ctypes.byref(gm), 0,
                                   ctypes.byref(st)), "de_gplmr_eig_d")
    if case["precision"] == "fp64":
        return {"e": e, "x": x}
    # A solve that is stopped at its tolerance defines the resonance energy;
    # the Ritz vector's phase is arbitrary and its direction is known to
    # about tol over the level spacing only.
    return {"e": e}


def work(case):
    nn, dim = 2 * case["n"] + 1, float(_dim(case))
    n = case["n"]

    def product(elem):
        """One H x: x read, y written; T commutes with the reflection of an
        axis, so a line of NN points takes (N+1)^2 + N^2 real-by-complex
        multiply-adds, and there are 6 NN^5 lines; then V x."""
        return 2 * elem * dim, 4.0 * 6 * nn ** 5 * ((n + 1) ** 2 + n ** 2) + 8 * dim

    if case["kind"] == "matvec":
        b, f = product(8 if case["storage"] == "c64" else 16)
        return {"bytes": case["nvec"] * b, "flops": case["nvec"] * f}
    if case["kind"] == "dots":
        return {"bytes": 16 * dim * (case["nbra"] + case["nket"]), "flops": 8 * dim * case["nbra"] * case["nket"]}
    # a solve: per outer iteration 1 + NS preconditioned blocks of 5 inner
    # products and one outer product each, and the projection, which reads
    # the (3 + NS) blocks and their products; a start converges in about 50
    its = case["maxit"] if case["precision"] == "fp64" else 50
    blocks, k = its * (1 + case["ns"]) * case["nev"], (3 + case["ns"]) * case["nev"]
    bo, fo = product(16)
    bi, fi = product(16 if case["precision"] == "fp64" else 8)
    return {"bytes": blocks * (bo + 5 * bi) + its * 2 * k * 16 * dim,
            "flops": blocks * (fo + 5 * fi) + its * 16 * k * k * dim}


# ---- the same values in 64 bits by plain numpy and torch

_INVERSE = {}


def _kinetic_row(d):
    """T(a, b) of the sinc-DVR second derivative at a - b = d."""
    d = np.asarray(d)
    with np.errstate(divide="ignore"):
        off = np.where(d % 2 == 0, 1.0, -1.0) / (DELTA ** 2 * d.astype(float) ** 2)
    return np.where(d == 0, (math.pi / DELTA) ** 2 / 6.0, off)


def _inverse_table(nout, nsmall=22, tfactor=4):
    """The regularised 1/r table on (-nout..nout)^3: delta^3/|r| on a big
    grid, corrected on a small one so that the kinetic operator applied to it
    is a point source."""
    if nout not in _INVERSE:
        nbig = nsmall * tfactor
        b, s = np.arange(-nbig, nbig + 1), np.arange(-nsmall, nsmall + 1)
        with np.errstate(divide="ignore"):
            r = DELTA ** 2 / np.sqrt(b[:, None, None] ** 2 + b[None, :, None] ** 2 + b[None, None, :] ** 2.0)
        r[nbig, nbig, nbig] = 0.0
        lo, hi = nbig - nsmall, nbig + nsmall + 1
        t = _kinetic_row(s[:, None] - b[None, :])
        along = np.einsum("ip,pjk->ijk", t, r[:, lo:hi, lo:hi], optimize=True)  # r is the same along every axis
        tr = -(along + along.transpose(1, 0, 2) + along.transpose(2, 1, 0))
        tr[nsmall, nsmall, nsmall] += 2 * math.pi
        w, v = np.linalg.eigh(_kinetic_row(s[:, None] - s[None, :]))
        q = np.einsum("ia,jb,kc,ijk->abc", v, v, v, tr, optimize=True)
        q = q / (w[:, None, None] + w[None, :, None] + w[None, None, :])
        r[lo:hi, lo:hi, lo:hi] += np.einsum("ia,jb,kc,abc->ijk", v, v, v, q, optimize=True)
        _INVERSE[nout] = r[nbig - nout:nbig + nout + 1, nbig - nout:nbig + nout + 1, nbig - nout:nbig + nout + 1].copy()
    return _INVERSE[nout]


def _potential(n):
    """V(r1, r2) times SCALE as an array (k2, j2, i2, k1, j1, i1)."""
    nn = 2 * n + 1
    table = torch.from_numpy(_inverse_table(nn)).cuda() / DELTA ** 3  # symmetric in its axes
    c = torch.arange(-n, n + 1, device="cuda") + nn
    near = table[c][:, c][:, :, c]
    d = torch.arange(nn, device="cuda")
    d = d[:, None] - d[None, :] + nn  # electron 2 minus electron 1
    k, j, i = (d.view([nn if a in (x, x + 3) else 1 for a in range(6)]) for x in range(3))
    v = table[k, j, i]
    v -= CHARGE * (near.view(nn, nn, nn, 1, 1, 1) + near.view(1, 1, 1, nn, nn, nn))
    return v


def _product(x, n, theta, v, t):
    nn = 2 * n + 1
    x = x.to(torch.complex128)
    kin = torch.matmul(x.view(-1, nn), t.to(torch.complex128))
    re = torch.view_as_real(x)
    out = torch.view_as_real(kin)
    for axis in range(5):  # the slower axes, one batch of real products each
        out.view(nn ** axis, nn, -1).add_(torch.matmul(t, re.view(nn ** axis, nn, -1)))
    kin = kin.view(-1) * complex(math.cos(2 * theta), -math.sin(2 * theta))
    return kin.add_(x * v.view(-1), alpha=complex(math.cos(theta), -math.sin(theta)))


def exact(case, seed):
    if case["kind"] == "solve":
        return None
    state = prepare(case, seed)
    if case["kind"] == "dots":
        bras = state["bras"].conj() if case["hermitian"] else state["bras"]
        return torch.stack([(bras * k).sum(dim=1) for k in state["kets"]])
    n, d = case["n"], np.arange(2 * case["n"] + 1)
    v, t = _potential(n), torch.from_numpy(_kinetic_row(d[:, None] - d[None, :])).cuda()
    del state["y"]
    return torch.stack([_product(x, n, case["theta"], v, t) for x in state["x"]])
