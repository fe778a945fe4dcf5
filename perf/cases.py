"""Performance cases: the eigensolves a program links this library for, through its public entry points.

Every case is one call (or one chain of calls) as a semi-empirical SCC program makes it: generalized solves on device
buffers, one per geometry; a factored solve per SCC cycle; the FP32 chain refined to FP64; the occupied orbitals only;
the refinement of the previous cycle's orbitals; uneven batches of molecules; the density-matrix adjoint; and the
host-pointer entries (LAPACK's dsygvd shape and the sytrd / stedc / ormtr chain that libxtb links).  Matrix orders run
from a few atoms (24) to the largest benchmark molecule (1788), odd ones among them.

Inputs: S = c I + G, G_ij = 0.35 exp(-|i-j|/12) u_ij (u uniform on [-1, 1]; c keeps the smallest eigenvalue near or above
0.05); eigenvalues spread over [-1.0, 0.5] Eh with level repulsion (a jittered lattice) and a 0.05 Eh HOMO/LUMO gap at
n/2; H = U^T Q diag(e) Q^T U with S = U^T U and Q a random orthogonal matrix, so that C = U^-1 Q.  Device work runs on
one stream that the program keeps.  Orbitals come back with the usual phase convention (the largest coefficient of an
orbital is positive), which makes them unique.
"""
from __future__ import annotations

import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xtb-diagonalization_b200")
for _p in (os.path.join(os.getcwd(), "xtb-diagonalization_b200"), _PKG):
    if os.path.isdir(_p) and _p not in sys.path:
        sys.path.append(_p)
import xtbeig  # noqa: E402

F64 = torch.float64
_stream = None


def _work_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ------------------------------------------------------------------------------------------------ cases


def listed():
    return [
        # The smallest calls: a molecule of a dozen atoms, where launches and latency are the whole cost.
        {"name": "sygvd_37", "kind": "sygvd", "n": 37, "m": 0, "precision": 64},
        # The lower end of the benchmark's uneven batch.
        {"name": "sygvd_130", "kind": "sygvd", "n": 130, "m": 0, "precision": 64},
        # The standard problem (an orthogonal basis) with a near-degenerate group.
        {"name": "syevd_412", "kind": "syevd", "n": 412},
        # One SCC cycle of a mid-size molecule: S was factored once per geometry.
        {"name": "factored_619", "kind": "factored", "n": 619, "precision": 64},
        # Occupied orbitals only, as an SCC cycle before convergence needs them.
        {"name": "lowest_1203", "kind": "sygvd", "n": 1203, "m": 601, "precision": 64},
        # The headline: every eigenpair of the largest benchmark molecule.
        {"name": "sygvd_1788", "kind": "sygvd", "n": 1788, "m": 0, "precision": 64},
        # The same through the FP32 chain with FP64 refinement (option "precision" = 32).
        {"name": "mixed_1788", "kind": "sygvd", "n": 1788, "m": 0, "precision": 32},
        # A late SCC cycle: the previous cycle's orbitals refined against the new H.
        {"name": "refine_1204", "kind": "refine", "n": 1204, "iters": 2},
        # A screening run: molecules of many sizes in one call.
        {"name": "batch_24", "kind": "batch", "count": 24, "lo": 124, "hi": 1788},
        # Gradients through the smeared density matrix (host arrays by the entry's nature).
        {"name": "adjoint_4x588", "kind": "adjoint", "n": 588, "count": 4, "temp": 300.0},
        # LAPACK's dsygvd from pinned host arrays: the drop-in whole solve.
        {"name": "host_776", "kind": "host", "n": 776, "uplo": "L"},
        # The chain libxtb links: dsytrd, dstedc and dormtr, each on host arrays.
        {"name": "dropin_412", "kind": "dropin", "n": 412},
    ]


def _log_n(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sygvd", "sygvd", "sygvd", "syevd", "factored", "refine", "batch", "adjoint", "host", "dropin"])
    if kind == "sygvd":
        n = _log_n(rng, 24, 1788)
        m = rng.choice([0, 0, max(1, n // 2 + rng.randint(-n // 8, n // 8))])
        return {"kind": kind, "n": n, "m": m, "precision": rng.choice([64, 64, 32])}
    if kind == "syevd":
        return {"kind": kind, "n": _log_n(rng, 24, 1204)}
    if kind == "factored":
        return {"kind": kind, "n": _log_n(rng, 24, 1788), "precision": rng.choice([64, 32])}
    if kind == "refine":
        return {"kind": kind, "n": _log_n(rng, 124, 1788), "iters": 2}
    if kind == "batch":
        lo = rng.randint(24, 400)
        return {"kind": kind, "count": rng.randint(6, 20), "lo": lo, "hi": rng.randint(lo + 100, 1500)}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_n(rng, 60, 588), "count": rng.randint(1, 6), "temp": rng.choice([300.0, 1000.0])}
    if kind == "host":
        return {"kind": kind, "n": _log_n(rng, 24, 1400), "uplo": rng.choice(["U", "L"])}
    return {"kind": kind, "n": _log_n(rng, 24, 900)}


def _batch_sizes(case):
    r = random.Random("%d %d %d" % (case["count"], case["lo"], case["hi"]))
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["count"])]


def work(case):
    """Bytes: the matrices the call reads and writes once (a symmetric input counts whole).  Flops: Cholesky n^3/3,
    congruence n^3, reduction 4n^3/3, tridiagonal eigensolve 4/3 n^2 m, back-transformations 2n^2 m and n^2 m."""

    def solve(n, m, general=True, factor=True):
        flops = (4 / 3) * n**3 + (4 / 3 + 2) * n * n * m
        if general:
            flops += n**3 + n * n * m + (n**3 / 3 if factor else 0)
        return flops

    kind = case["kind"]
    if kind == "batch":
        ns = _batch_sizes(case)
        return {"bytes": sum(8 * (4 * n * n + n) for n in ns), "flops": sum(solve(n, n) for n in ns)}
    n = case["n"]
    nn = n * n
    if kind == "sygvd":
        m = case["m"] or n
        return {"bytes": 8 * (3 * nn + n * m + n), "flops": solve(n, m)}
    if kind == "syevd":
        return {"bytes": 8 * (2 * nn + n), "flops": solve(n, n, general=False)}
    if kind == "factored":
        return {"bytes": 8 * (4 * nn + n), "flops": solve(n, n, factor=False)}
    if kind == "refine":
        return {"bytes": 8 * (4 * nn + n), "flops": case["iters"] * 8.0 * n**3}
    if kind == "adjoint":
        return {"bytes": case["count"] * 8 * 5 * nn, "flops": case["count"] * (solve(n, n) + 12.0 * n**3)}
    if kind == "host":
        return {"bytes": 8 * (4 * nn + n), "flops": solve(n, n)}
    return {"bytes": 8 * (6 * nn + 4 * n), "flops": solve(n, n, general=False)}


# ------------------------------------------------------------------------------------------------ inputs


def _spectrum(n, gen, gap):
    jitter = (torch.rand(n, generator=gen, device="cuda", dtype=F64) - 0.5) * 0.7
    e = -1.0 + 1.5 * (torch.arange(n, device="cuda", dtype=F64) + 0.5 + jitter) / n
    if gap:
        e[n // 2:] += 0.05
    return e


def _orthogonal(n, gen):
    q, r = torch.linalg.qr(torch.randn(n, n, generator=gen, device="cuda", dtype=F64))
    return q * torch.sign(torch.diagonal(r))[None, :]


def _pair(n, gen):
    """(H, S, C) with H C = S C diag(e), C^T S C = I, e ascending (all n x n, on the GPU)."""
    i = torch.arange(n, device="cuda", dtype=F64)
    u = torch.rand(n, n, generator=gen, device="cuda", dtype=F64) * 2 - 1
    g = torch.triu(0.35 * torch.exp(-(i[:, None] - i[None, :]).abs() / 12.0) * u, 1)
    g = g + g.T
    v = torch.randn(n, 1, generator=gen, device="cuda", dtype=F64)
    for _ in range(24):  # the norm of G, from below
        v = g @ v
        norm = torch.linalg.vector_norm(v)
        v = v / norm
    s = g + torch.clamp(1.1 * norm + 0.05, min=1.0) * torch.eye(n, device="cuda", dtype=F64)
    upper = torch.linalg.cholesky(s, upper=True)
    e = _spectrum(n, gen, True)
    q = _orthogonal(n, gen)
    uq = upper.T @ q
    h = (uq * e[None, :]) @ uq.T
    return (0.5 * (h + h.T)).contiguous(), s.contiguous(), upper, q


def _standard(n, gen):
    """A symmetric matrix with a near-degenerate group of eight eigenvalues."""
    e = _spectrum(n, gen, False)
    if n >= 64:
        e[n // 3: n // 3 + 8] = e[n // 3] + 1e-5 * torch.arange(8, device="cuda", dtype=F64)
    q = _orthogonal(n, gen)
    a = (q * e[None, :]) @ q.T
    return (0.5 * (a + a.T)).contiguous()


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _perturbed(h, n, gen):
    r = torch.randn(n, n, generator=gen, device="cuda", dtype=F64)
    return (h + 2.5e-7 * (r + r.T)).contiguous()


def _inputs(case, seed):
    """What the call computes from, on the GPU (symmetric matrices: row-major is column-major)."""
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "batch":
        return [_pair(n, gen)[:2] for n in _batch_sizes(case)]
    n = case["n"]
    if kind in ("syevd", "dropin"):
        return (_standard(n, gen),)
    if kind == "refine":
        h, s, upper, q = _pair(n, gen)
        c = torch.linalg.solve_triangular(upper, q, upper=True)
        return _perturbed(h, n, gen), s, c.T.contiguous()
    if kind == "adjoint":
        out = []
        for _ in range(case["count"]):
            h, s = _pair(n, gen)[:2]
            w = torch.randn(n, n, generator=gen, device="cuda", dtype=F64)
            out.append((h, s, 0.5 * (w + w.T)))
        return out
    return _pair(n, gen)[:2]


KB = 3.166808578545117e-06  # Eh / K


def _mid_gap(n):
    """The chemical potential of the half-filled band: between the lattice sites n/2 - 1 and n/2."""
    return -1.0 + 1.5 * (n // 2) / n + 0.025


def prepare(case, seed):
    kind = case["kind"]
    xtbeig.set_option("precision", case.get("precision", 64))
    stream = _work_stream()
    x = _inputs(case, seed)
    st = {"case": dict(case), "stream": stream, "handle": stream.cuda_stream}
    if kind == "batch":
        ns = _batch_sizes(case)
        total = sum(n * n for n in ns)
        st["ns"] = ns
        for key, at in (("h0", 0), ("s0", 1)):
            st[key] = torch.cat([p[at].reshape(-1) for p in x])
        st["h"], st["s"] = torch.empty_like(st["h0"]), torch.empty_like(st["s0"])
        st["w"] = torch.empty(sum(ns), device="cuda", dtype=F64)
        assert st["h"].numel() == total
        off = woff = 0
        st["hv"], st["hp"], st["sp"], st["wp"] = [], [], [], []
        for n in ns:
            st["hv"].append(st["h"][off: off + n * n].view(n, n))
            st["hp"].append(st["h"].data_ptr() + 8 * off)
            st["sp"].append(st["s"].data_ptr() + 8 * off)
            st["wp"].append(st["w"].data_ptr() + 8 * woff)
            off += n * n
            woff += n
    elif kind == "adjoint":
        st["kt"] = [KB * case["temp"]] * case["count"]
        st["mu"] = [_mid_gap(case["n"])] * case["count"]
        st["hs"], st["ss"], st["ws"] = (
            [np.asfortranarray(p[k].cpu().numpy()) for p in x] for k in range(3))
    elif kind == "host":
        st["h0"], st["s0"] = (p.cpu() for p in x)
        st["h"], st["s"] = (torch.empty_like(p).pin_memory() for p in (st["h0"], st["s0"]))
        st["w"] = torch.empty(case["n"], dtype=F64).pin_memory()
    elif kind == "dropin":
        n = case["n"]
        st["a0"] = x[0].cpu().numpy().T
        st["a"], st["z"] = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")
        st["d"], st["e"], st["tau"] = np.zeros(n), np.zeros(n), np.zeros(n)
        st["iwork"] = np.zeros(3 + 5 * n, np.int32)
        st["work"] = np.zeros(max(1 + 4 * n + n * n, 32 * (4 * n + 32)))
    else:
        n = case["n"]
        st["w"] = torch.empty(n, device="cuda", dtype=F64)
        st["h0"] = x[0]
        st["h"] = torch.empty_like(x[0])
        if kind == "factored":
            u, inv = x[1].clone(), torch.empty_like(x[1])
            torch.cuda.synchronize()
            _check(xtbeig.dsygvd_factor_device(n, u.data_ptr(), n, inv.data_ptr(), n, st["handle"]))
            st["u"], st["x"] = u, inv
        elif kind == "refine":
            st["s0"], st["c0"], st["c"] = x[1], x[2], torch.empty_like(x[2])
        elif kind == "sygvd":
            st["s0"], st["s"] = x[1], torch.empty_like(x[1])
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------------------------------------ the calls


def _check(info):
    if info != 0:
        raise RuntimeError("info %d: %s" % (info, xtbeig.last_error()))


def _phase(c):
    """Orbitals (rows) with their largest coefficient positive, in place."""
    big = torch.gather(c, 1, c.abs().argmax(dim=1, keepdim=True))
    return c.mul_(torch.sign(big))


def _phase_np(c):
    """The same for the columns of a host array."""
    big = c[np.abs(c).argmax(axis=0), np.arange(c.shape[1])]
    c *= np.sign(big)[None, :]
    return c


def _as_c_int(v):
    return ctypes.byref(ctypes.c_int(v))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "adjoint":
        dh, ds, info = xtbeig.density_adjoint_batched(st["hs"], st["ss"], st["kt"], st["mu"], st["ws"])
        return {"dh": dh, "ds": ds, "info": info}
    n = case.get("n", 0)
    if kind == "host":
        st["h"].copy_(st["h0"])
        st["s"].copy_(st["s0"])
        info = ctypes.c_int(0)
        one = _as_c_int(1)
        # The arrays are symmetric, so the row-major tensors are the column-major matrices.
        xtbeig.lib().xtb_dsygvd_gpu(one, b"V", case["uplo"].encode(), _as_c_int(n), ctypes.c_void_p(st["h"].data_ptr()),
                                    _as_c_int(n), ctypes.c_void_p(st["s"].data_ptr()), _as_c_int(n),
                                    ctypes.c_void_p(st["w"].data_ptr()), None, one, None, one, ctypes.byref(info))
        _check(info.value)
        return {"w": st["w"], "c": _phase(st["h"]), "u": st["s"]}
    if kind == "dropin":
        a, z, d, e, tau = st["a"], st["z"], st["d"], st["e"], st["tau"]
        np.copyto(a, st["a0"])
        xtbeig.xtb_dsytrd_upper(n, a, n, d, e, tau, st["work"])
        _check(xtbeig.xtb_dstedc(n, d, e, z, n, st["work"], 1 + 4 * n + n * n, st["iwork"], 3 + 5 * n))
        xtbeig.xtb_dormtr_upper(n, n, a, n, tau, z, n, st["work"])
        return {"w": d, "c": _phase_np(z)}
    with torch.cuda.stream(st["stream"]):
        st["h"].copy_(st["h0"])
        if kind == "batch":
            st["s"].copy_(st["s0"])
            info, ret = xtbeig.dsygvd_batched_device(st["ns"], st["hp"], st["ns"], st["sp"], st["ns"], st["wp"],
                                                     st["handle"])
            _check(ret)
            for c in st["hv"]:
                _phase(c)
            return {"w": st["w"], "c": st["h"], "u": st["s"], "info": info}
        h, w = st["h"], st["w"]
        if kind == "syevd":
            _check(xtbeig.dsyevd_device(n, h.data_ptr(), n, w.data_ptr(), st["handle"]))
            return {"w": w, "c": _phase(h)}
        if kind == "factored":
            _check(xtbeig.dsygvd_factored_device(n, h.data_ptr(), n, st["u"].data_ptr(), n, st["x"].data_ptr(), n,
                                                 w.data_ptr(), st["handle"]))
            return {"w": w, "c": _phase(h)}
        if kind == "refine":
            c = st["c"].copy_(st["c0"])
            _check(xtbeig.dsygvd_refine_device(n, h.data_ptr(), n, st["s0"].data_ptr(), n, c.data_ptr(), n,
                                               w.data_ptr(), case["iters"], st["handle"]))
            return {"w": w, "c": _phase(c)}
        st["s"].copy_(st["s0"])
        m = case["m"]
        if m:
            _check(xtbeig.dsygvd_lowest_device(n, m, h.data_ptr(), n, st["s"].data_ptr(), n, w.data_ptr(),
                                               st["handle"]))
            # The eigenvalues beyond the wanted ones (and a margin) are the FP32 chain's at precision 32.
            return {"w": w[:m] if case["precision"] == 32 else w, "c": _phase(h[:m]), "u": st["s"]}
        _check(xtbeig.dsygvd_device(n, h.data_ptr(), n, st["s"].data_ptr(), n, w.data_ptr(), st["handle"]))
        return {"w": w, "c": _phase(h), "u": st["s"]}


# ------------------------------------------------------------------------------------------------ 64-bit values


def _exact_pair(h, s, m=0):
    """(w, orbitals as rows, U in the column-major upper triangle with S's other triangle) of one pair."""
    low = torch.linalg.cholesky(s)
    a = torch.linalg.solve_triangular(low, h, upper=False)
    a = torch.linalg.solve_triangular(low, a.T.contiguous(), upper=False)
    w, z = torch.linalg.eigh(0.5 * (a + a.T))
    c = _phase(torch.linalg.solve_triangular(low.T, z, upper=True).T.contiguous())
    return w, (c[:m] if m else c), torch.tril(low) + torch.triu(s, 1)


def _exact_adjoint(h, s, wbar, kt, mu):
    """Gradients of sum(wbar o P), P = C f(e) C^T, by the Daleckii-Krein formula."""
    e, c, _ = _exact_pair(h, s)
    c = c.T
    x = (e - mu) / kt
    sig = 1.0 / (1.0 + torch.exp(x.clamp(-700.0, 700.0)))
    a, b = x[:, None], x[None, :]
    half = 0.5 * (a - b)
    ch = torch.cosh((0.5 * x).clamp(-350.0, 350.0))
    series = -(1.0 + half**2 / 6 + half**4 / 120) / (4 * ch[:, None] * ch[None, :])
    diff = torch.where(a == b, torch.ones_like(half), a - b)
    ds = torch.where(half.abs() < 1e-2, series, (sig[:, None] - sig[None, :]) / diff)
    d1 = (2.0 / kt) * ds
    f = 2.0 * sig
    d2 = 0.5 * (f[:, None] + f[None, :]) + 0.5 * (e[:, None] + e[None, :]) * d1
    wh = c.T @ wbar @ c
    gh, gs = c @ (wh * d1) @ c.T, -(c @ (wh * d2) @ c.T)
    return 0.5 * (gh + gh.T), 0.5 * (gs + gs.T)


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "batch":
        parts = [_exact_pair(h, s) for h, s in x]
        w, c, u = (torch.cat([p[k].reshape(-1) for p in parts]) for k in range(3))
        return {"w": w, "c": c, "u": u, "info": None}
    n = case["n"]
    if kind == "adjoint":
        parts = [_exact_adjoint(h, s, wb, KB * case["temp"], _mid_gap(n)) for h, s, wb in x]
        return {"dh": [p[0].cpu().numpy() for p in parts], "ds": [p[1].cpu().numpy() for p in parts], "info": None}
    if kind in ("syevd", "dropin"):
        w, z = torch.linalg.eigh(x[0])
        c = _phase(z.T.contiguous())
        return {"w": w, "c": c} if kind == "syevd" else {"w": w.cpu().numpy(), "c": c.T.contiguous().cpu().numpy()}
    if kind == "host":
        w, c, u = _exact_pair(*x)
        if case["uplo"] == "L":  # the factor in the column-major lower triangle
            u = torch.tril(x[1], -1) + torch.linalg.cholesky(x[1]).T
        return {"w": w.cpu(), "c": c.cpu(), "u": u.cpu()}
    m = case.get("m", 0)
    w, c, u = _exact_pair(x[0], x[1], m)
    if kind == "sygvd":
        return {"w": w[:m] if m and case["precision"] == 32 else w, "c": c, "u": u}
    return {"w": w, "c": c}
