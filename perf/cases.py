"""The calls that a user of the framework makes, at the sizes they are made at.

A GNOF energy is an alternation of orbital steps (rotation, Lagrangian, packed
gradient, update) and occupation solves (J_MO, K_MO, H_core on the device, a CG
on the host), on an RI tensor b[m, n, l] that stays on the GPU.  So the cases
are the two contractions that every iteration makes (the Lagrangian and
JKH_MO), the optimiser loop around the first, the per-call pattern of a host
program that drives it (rotate_orbital and compute_Lagrange2 with host arrays),
the grouped loop over several molecules, the energy loop itself, the mixed form
of the Lagrangian, and the RI tensor from the integrals that precedes them all.

Sizes are the framework's workloads: (H2O)_k and alkanes in a double-zeta basis
with a fitting set (nbf = 24k, naux = 116k, nbf5 = 20k; n-octane 202 / 974 / 198)
and the synthetic 256 / 1024 / 64.  The FP64 form's first contraction runs from
digit slices (set_fp64_tc) from nbf = 128 on, as the server chooses, else on the
FP64 GEMM.  b, C and H have the distributions of donof_b200.workload.

A CUDA array of the framework holds Julia's column-major memory, so a tensor's
indices here run in reverse: b[l, n, m], C[p, m], elag[b, a].
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("donof.jl_b200"))
import donof_b200 as d  # noqa: E402
from donof_b200 import api, gnof, integrals, workload  # noqa: E402

TC_MIN_NBF = 128  # the server's rule for the digit slices
METHODS = ("ADAM", "ADABelief", "YOGI", "Demon")


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one water molecule: the smallest molecule anyone runs, bound by launches
        dict(name="lagrange-water", kind="lagrange", nbf=24, naux=116, nbeta=5, ncwo=3, open=0),
        # a radical in an odd-sized basis: open shell, ragged tiles, rows that are not 16-byte aligned
        dict(name="lagrange-radical", kind="lagrange", nbf=91, naux=437, nbeta=11, ncwo=5, open=2),
        # n-octane, the Lagrangian of an ordinary molecule with every orbital active
        dict(name="lagrange-octane", kind="lagrange", nbf=202, naux=974, nbeta=33, ncwo=5, open=0),
        # sixteen waters: the largest molecule of the served range
        dict(name="lagrange-water16", kind="lagrange", nbf=384, naux=1856, nbeta=80, ncwo=3, open=0),
        # the benchmark's orbital optimisation: ten iterations of one call
        dict(name="orbopt-256", kind="orbopt", nbf=256, naux=1024, nbeta=16, ncwo=3, open=0, method="ADAM", maxloop=10),
        # one iteration driven from host arrays, as DoNOF.jl's loop drives its GPU plugin
        dict(name="hoststep-256", kind="hoststep", nbf=256, naux=1024, nbeta=16, ncwo=3, open=0),
        # what each occupation solve takes from the device, eight waters
        dict(name="jkh-water8", kind="jkh", nbf=192, naux=928, nbeta=40, ncwo=3, open=0),
        # the mixed form where the fused kernel takes it, and where the general pipeline does
        dict(name="mixed-256", kind="mixed", nbf=256, naux=1024, nbeta=16, ncwo=3, open=0),
        dict(name="mixed-octane", kind="mixed", nbf=202, naux=974, nbeta=33, ncwo=5, open=0),
        # a batch of uneven water clusters advanced together
        dict(name="batch-water", kind="batch", count=16, kmax=8, maxloop=5),
        # whole call: three outer iterations of the energy of four waters
        dict(name="energy-water4", kind="energy", nbf=96, naux=464, nbeta=20, ncwo=3, open=0, maxit=3),
        # whole call: the RI tensor of eight waters from its integrals, and its first use
        dict(name="iaux-water8", kind="iaux", waters=8),
    ]


def _sizes(rng, lo, hi):
    nbf = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    nbf += rng.choice((0, 0, 1, 3))
    ncwo = rng.randint(1, 5)
    nopen = rng.choice((0, 0, 0, 1, 2))
    most = max(1, (nbf - nopen) // (1 + ncwo))
    nbeta = max(1, int(most * rng.uniform(0.25, 1.0)))
    return dict(nbf=nbf, naux=int(nbf * rng.uniform(3.0, 5.0)) + 1, nbeta=nbeta, ncwo=ncwo, open=nopen)


def draw(rng):
    kind = rng.choice(("lagrange", "lagrange", "lagrange", "orbopt", "hoststep", "jkh", "jkh", "mixed", "mixed",
                       "batch", "energy", "iaux"))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), kmax=rng.randint(2, 8), maxloop=rng.randint(2, 5))
    if kind == "iaux":
        return dict(kind=kind, waters=rng.randint(1, 7))
    if kind == "energy":
        return dict(kind=kind, maxit=rng.randint(1, 3), **_sizes(rng, 24, 96))
    if kind == "orbopt":
        return dict(kind=kind, method=rng.choice(METHODS), maxloop=rng.randint(2, 10), **_sizes(rng, 24, 256))
    return dict(kind=kind, **_sizes(rng, 24, 300 if kind == "hoststep" else 380))


# ---------------------------------------------------------------- inputs
def _ctx():
    return d.default_context()


def _nbf5(c):
    return c["nbeta"] * (1 + c["ncwo"]) + c["open"]


def _dev(a):
    return d.to_device(a)


class Job:
    """A molecule as a program holds it: b on the GPU, the arrays of the functional."""

    def __init__(self, c, seed, precision="fp64"):
        wl = workload.synthetic(nbf=c["nbf"], naux=c["naux"], nbeta=c["nbeta"], ncwo=c["ncwo"], seed=seed, with_b=False)
        self.p, self.Ch, self.Hh = wl.p, wl.C, wl.H
        self.nh, self.cjh, self.ckh = wl.n, wl.cj12, wl.ck12
        if c["open"]:
            self.p = d.Param(nbf=c["nbf"], nbfaux=c["naux"], nbeta=c["nbeta"], nalpha=c["nbeta"] + c["open"], ncwo=c["ncwo"])
            gamma = np.random.default_rng(seed + 5).standard_normal(self.p.nv)
            self.nh, _ = gnof.occupations(gamma, self.p)
            self.cjh, self.ckh = (np.asfortranarray(x) for x in gnof.coupling(self.nh, self.p))
        self.C, self.H, self.n, self.cj, self.ck = (_dev(x) for x in (self.Ch, self.Hh, self.nh, self.cjh, self.ckh))
        self.raw = workload.b_device(c["nbf"], c["naux"], seed)
        self.b = d.eris_to_gpu(self.raw, precision, _ctx())
        if precision == "fp64" and c["nbf"] >= TC_MIN_NBF:
            self.b.set_fp64_tc(True)


def _empty(*shape):
    return torch.empty(shape, dtype=torch.float64, device="cuda")


def _water_integrals(c, seed):
    orb, aux = workload.water_cluster_bases(c["waters"], seed=seed)
    G = integrals.ERI_2e2c(aux)
    G = np.asfortranarray((G + G.T) / 2)
    t = integrals.ERI_2e3c_dev(orb, aux, _ctx())
    I = t.cpu().numpy().reshape((orb.nbas, orb.nbas, aux.nbas), order="F")
    Q = np.linalg.qr(np.random.default_rng(seed).standard_normal((orb.nbas, orb.nbas)))[0]
    return G, I, np.asfortranarray(Q), 20 * c["waters"]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("lagrange", "mixed", "jkh", "orbopt", "hoststep"):
        j = s["job"] = Job(case, seed, "mixed" if kind == "mixed" else "fp64")
        nbf, nbf5 = case["nbf"], _nbf5(case)
        if kind in ("lagrange", "mixed"):
            s["elag"], s["Hmat"], s["E"] = _empty(nbf, nbf), _empty(nbf5, nbf), _empty(1)
        elif kind == "jkh":
            s["J"], s["K"], s["Hc"] = _empty(nbf5, nbf5), _empty(nbf5, nbf5), _empty(nbf5)
        elif kind == "hoststep":
            def pinned(a):
                h = d.host_pinned(a.shape)
                h[...] = a
                return h
            s["y"] = pinned(0.01 * np.random.default_rng(seed + 1).standard_normal(j.p.nvar))
            s["host"] = [pinned(np.asfortranarray(x)) for x in (j.Ch, j.nh, j.Hh, j.cjh, j.ckh)]
            s["Cn"], s["elag"], s["Hmat"] = (d.host_pinned(x) for x in ((nbf, nbf), (nbf, nbf), (nbf, nbf5)))
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        ks = np.sort(rng.permutation(np.arange(case["count"]) % case["kmax"] + 1))[::-1]  # every size of the range
        jobs = s["jobs"] = [Job(_water(int(k)), 1000 * seed + i) for i, k in enumerate(ks)]
        s["batch"] = d.Batch([j.b for j in jobs], [j.p for j in jobs], _ctx())
    elif kind == "energy":
        p = d.Param(nbf=case["nbf"], nbfaux=case["naux"], nbeta=case["nbeta"], nalpha=case["nbeta"] + case["open"],
                    ncwo=case["ncwo"])
        wl = workload.molecule_like(nbf=case["nbf"], naux=case["naux"], nbeta=case["nbeta"], ncwo=case["ncwo"], seed=seed)
        s["p"], s["H"], s["C"], s["gamma"] = p, wl.H, wl.C, gnof.guess_gamma(p)
        s["b"] = d.eris_to_gpu(wl.b, "fp64", _ctx())
        if case["nbf"] >= TC_MIN_NBF:
            s["b"].set_fp64_tc(True)
    elif kind == "iaux":
        s["G"], s["I"], C, s["nbf5"] = _water_integrals(case, seed)
        s["C"] = _dev(C)
        s["out"] = _empty(s["G"].shape[0], s["nbf5"], s["nbf5"])
    return s


def _water(k):
    return dict(nbf=24 * k, naux=116 * k, nbeta=5 * k, ncwo=3, open=0)


# ---------------------------------------------------------------- one pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    j = s.get("job")
    if kind in ("lagrange", "mixed"):
        d.compute_Lagrange2_dev(j.C, j.n, j.H, j.b, j.cj, j.ck, j.p.nalpha, j.p.nbeta, s["elag"], s["Hmat"], s["E"])
        return {"elag": s["elag"], "Hmat": s["Hmat"], "E": s["E"]}
    if kind == "jkh":
        d.JKH_MO_dev(j.C, j.H, j.b, _nbf5(c), s["J"], s["K"], s["Hc"])
        return {"J": s["J"], "K": s["K"], "Hc": s["Hc"]}
    if kind == "orbopt":
        C = j.C.clone()
        E, nit, ok, alpha, maxloop = d.orbopt_dev(c["method"], j.n, j.cj, j.ck, j.H, C, j.b, j.p, 0.01, c["maxloop"],
                                                  j.p.threshgorb)
        return {"E": E, "C": C, "nit": nit, "ok": ok, "alpha": alpha, "maxloop": maxloop}
    if kind == "hoststep":
        C, n, H, cj, ck = s["host"]
        Cn = d.rotate_orbital(s["y"], C, j.p, _ctx(), out=s["Cn"])
        elag, Hmat, E = d.compute_Lagrange2(Cn, n, H, j.b, cj, ck, j.p.nalpha, j.p.nbeta, return_energy=True,
                                            out=(s["elag"], s["Hmat"]))
        return {"C": Cn, "elag": elag, "Hmat": Hmat, "E": E}
    if kind == "batch":
        jobs, k = s["jobs"], len(s["jobs"])
        C = [x.C.clone() for x in jobs]
        got = s["batch"].orbopt("ADAM", [x.n for x in jobs], [x.cj for x in jobs], [x.ck for x in jobs],
                                [x.H for x in jobs], C, [0.01] * k, [c["maxloop"]] * k, [x.p.threshgorb for x in jobs])
        return {"E": torch.tensor([g[0] for g in got], dtype=torch.float64), "nit": torch.tensor([g[1] for g in got]), "C": C}
    if kind == "energy":
        p = d.Param(nbf=c["nbf"], nbfaux=c["naux"], nbeta=c["nbeta"], nalpha=c["nbeta"] + c["open"], ncwo=c["ncwo"])
        C, gamma, n, elag, res, _ = api.energy_loop(s["H"], s["b"], p, s["C"], s["gamma"], maxit=c["maxit"])
        return {"C": C, "gamma": gamma, "n": n, "elag": elag, "E": res["E_elec"], "iterations": res["iterations"]}
    b = d.Iaux_gpu(s["G"], s["I"], "fp64", _ctx())
    d.transform_dev(s["C"], b, s["nbf5"], out=s["out"])
    b.free()
    return s["out"]


# ---------------------------------------------------------------- what a pass cannot do without
def _steps(c):
    """bytes and flops of the three contractions and the tail of one Lagrangian."""
    nbf, naux, nbf5 = c["nbf"], c["naux"], _nbf5(c)
    b = 8.0 * nbf * nbf * naux
    t1, t2 = 2.0 * nbf * nbf * nbf5 * naux, 2.0 * nbf * nbf5 * nbf5 * naux
    tail = 2.0 * nbf * nbf * nbf5 * 3
    small = 8.0 * (3 * nbf * nbf + nbf * nbf5 + 2 * nbf5 * nbf5)
    return b, small, t1, t2, tail


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = [work(dict(kind="orbopt", maxloop=case["maxloop"], **_water(k % case["kmax"] + 1))) for k in range(case["count"])]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    if kind == "iaux":
        k = case["waters"]
        nbf, naux, nbf5 = 24 * k, 64 * k, 20 * k
        return {"bytes": 8.0 * (nbf * nbf * naux + naux * naux + nbf5 * nbf5 * naux),
                "flops": 2.0 * nbf * nbf * naux * naux + 9.0 * naux ** 3 + 2.0 * nbf * nbf5 * (nbf + nbf5) * naux}
    b, small, t1, t2, tail = _steps(case)
    rot = 2.0 * case["nbf"] ** 3 * 8
    if kind == "lagrange":
        return {"bytes": b + small, "flops": t1 + 2 * t2 + tail}
    if kind == "mixed":
        return {"bytes": b / 2 + small, "flops": t1 + 2 * t2 + tail}
    if kind == "jkh":
        return {"bytes": b + small, "flops": t1 + t2}
    if kind == "hoststep":
        return {"bytes": b + 2 * small, "flops": t1 + 2 * t2 + tail + rot}
    if kind == "orbopt":
        n = case["maxloop"]
        return {"bytes": (n + 1) * (b + small), "flops": (n + 1) * (t1 + 2 * t2 + tail) + n * rot}
    n = case["maxit"]
    return {"bytes": n * (12 * b + 11 * small), "flops": n * (12 * (t1 + 2 * t2 + tail) + 10 * rot)}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch
def _transform(C5, b):
    tmp = torch.matmul(C5, b)                 # [l, q, m]
    return tmp, torch.matmul(tmp, C5.T)       # [l, q, p]


def _chunks(b, most=2 ** 26):
    step = max(1, most // (b.shape[1] * b.shape[2]))
    return (b[i:i + step] for i in range(0, b.shape[0], step))


def _lagrange(C, n, H, b, cj, ck, nalpha, nbeta):
    nbf5 = n.shape[0]
    C5 = C[:nbf5]
    at = torch.arange(nbf5, device=C.device)
    occ = torch.where((at < nbeta) | (at >= nalpha), n, torch.zeros_like(n)) if nbeta > 0 else torch.zeros_like(n)
    Y = torch.zeros_like(C5)
    for part in _chunks(b):
        tmp, bpq = _transform(C5, part)
        diag = torch.diagonal(bpq, dim1=1, dim2=2)
        W = -ck * bpq                         # [l, q, b]
        torch.diagonal(W, dim1=1, dim2=2).add_(occ * diag + diag @ cj)
        Y += torch.matmul(W.reshape(-1, nbf5).T, tmp.reshape(-1, C.shape[1]))
    Hmat = (C5 @ H) @ C.T                     # [b, a]
    elag = torch.zeros_like(H)
    elag[:nbf5] = n[:, None] * Hmat + Y @ C.T
    E = (torch.diagonal(elag)[:nbf5] + n * torch.diagonal(Hmat)).sum()
    return elag, Hmat, E


def _rotate(y, C, nbf5):
    nbf = C.shape[0]
    i, j = torch.triu_indices(nbf5, nbf, 1, device=C.device)
    Y = torch.zeros_like(C)
    Y[i, j] = y
    Y[j, i] = -y
    return torch.matrix_exp(Y).T @ C          # (C U)^T


def _orbopt(method, C, n, H, b, cj, ck, p, alpha, maxloop):
    elag, Hmat, E = _lagrange(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    i, j = torch.triu_indices(p.nbf5, p.nbf, 1, device=C.device)
    beta1, beta2 = (0.6, 0.999) if method == "Demon" else (0.5, 0.9)
    first = beta1
    m = v = vmax = torch.zeros(i.shape[0], dtype=torch.float64, device=C.device)
    best, nit, ok, improved = (float(E), C), 0, False, False
    loops = maxloop
    for it in range(1, maxloop + 1):
        nit += 1
        g = 4.0 * (elag[j, i] - elag[i, j])   # elag[a, b] is stored [b, a]
        if 2.0 * float(g.abs().max()) < p.threshgorb and improved:
            ok = True
            break
        if method == "Demon":
            rate = (it - 1.0) / (maxloop - 1.0)
            beta1 = first * (1.0 - rate) / ((1.0 - first) + first * (1.0 - rate))
        m = beta1 * m + (1.0 - beta1) * g
        if method == "ADABelief":
            v = beta2 * v + (1.0 - beta2) * (g - m) ** 2
        elif method == "YOGI":
            v = v - (1.0 - beta2) * torch.sign(v - g * g) * g * g
        else:
            v = beta2 * v + (1.0 - beta2) * g * g
        vmax = torch.maximum(vmax, v / (1.0 - beta2 ** it))
        y = -alpha * (m / (1.0 - beta1 ** it)) / torch.sqrt(vmax + 1e-16)
        C = _rotate(y, C, p.nbf5)
        elag, Hmat, E = _lagrange(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
        if float(E) < best[0]:
            best, improved = (float(E), C), True
    if not improved:
        alpha, loops = 0.3 * alpha, maxloop + 10
    E, C = best if loops < 100 else (float(E), C)
    return {"E": E, "C": C, "nit": nit, "ok": ok, "alpha": alpha, "maxloop": loops}


def exact(case, seed):
    kind = case["kind"]
    if kind == "energy":  # its occupation solver has no counterpart in torch or numpy
        return None
    if kind == "iaux":
        G, I, C, nbf5 = _water_integrals(case, seed)
        nbf, naux = I.shape[0], I.shape[2]
        w, V = torch.linalg.eigh(torch.from_numpy(np.ascontiguousarray(G)).cuda())
        s = torch.where(w < 0, torch.zeros_like(w), 1.0 / torch.sqrt(w.abs()))
        It = torch.from_numpy(np.ascontiguousarray(I.T)).cuda().reshape(naux, nbf * nbf)
        b = (((V * s) @ V.T) @ It).reshape(naux, nbf, nbf)
        return _transform(_dev(C)[:nbf5], b)[1]
    if kind == "batch":
        s = prepare(case, seed)
        got = [_orbopt("ADAM", j.C, j.n, j.H, j.raw, j.cj, j.ck, j.p, 0.01, case["maxloop"]) for j in s["jobs"]]
        return {"E": torch.tensor([g["E"] for g in got], dtype=torch.float64), "nit": torch.tensor([g["nit"] for g in got]),
                "C": [g["C"] for g in got]}
    j = Job(case, seed, "mixed" if kind == "mixed" else "fp64")
    p = j.p
    if kind in ("lagrange", "mixed"):
        elag, Hmat, E = _lagrange(j.C, j.n, j.H, j.raw, j.cj, j.ck, p.nalpha, p.nbeta)
        return {"elag": elag, "Hmat": Hmat, "E": E.reshape(1)}
    if kind == "orbopt":
        return _orbopt(case["method"], j.C, j.n, j.H, j.raw, j.cj, j.ck, p, 0.01, case["maxloop"])
    if kind == "jkh":
        C5 = j.C[:p.nbf5]
        J = torch.zeros(p.nbf5, p.nbf5, dtype=torch.float64, device="cuda")
        K = torch.zeros_like(J)
        for part in _chunks(j.raw):
            bpq = _transform(C5, part)[1]
            diag = torch.diagonal(bpq, dim1=1, dim2=2)
            J += diag.T @ diag
            K += (bpq * bpq).sum(0)
        return {"J": J, "K": K, "Hc": ((C5 @ j.H) * C5).sum(1)}
    y = torch.from_numpy(0.01 * np.random.default_rng(seed + 1).standard_normal(p.nvar)).cuda()
    C = _rotate(y, j.C, p.nbf5)
    elag, Hmat, E = _lagrange(C, j.n, j.H, j.raw, j.cj, j.ck, p.nalpha, p.nbeta)
    up = lambda t: t.T.cpu().numpy()  # noqa: E731  (host arrays are indexed like Julia's)
    return {"C": up(C), "elag": up(elag), "Hmat": up(Hmat), "E": float(E)}
