"""What the digits of csrc/ozaki.cu keep of elements of very different size, restated on
the CPU with exact integers: an RI tensor whose basis functions differ by many decades (a
tight function beside a diffuse one, fragments of unlike scale), orbitals that do not mix
them or that are not normalised, and a molecule's integrals.  Every element of b_pq, elag,
J and K has a bound of its own; the scales hold it while the row norms of b are within
ROW_SPREAD = 64, and do not beyond, where T2 and Y run as FP64 GEMMs of T1's tmp.

Bounds.  T1's operands are truncated to 49 bits below a power of two that is at most
twice the largest element of the row of b_l (D[m, l]) or of the column of C5 (c[q]), and
the digit products from i + j = 7 on are left out: (2^-48 + 2^-48 + 28 2^-49) D c for
each of the nbf products, so |d tmp[m, q, l]| <= nbf 2^-44 D[m, l] c[q].  The later
contractions hold their operands to 2^-56 of the same sizes, which twice the bound
covers; it is carried through b_pq, W, Y, elag, J and K with absolute values.
"""
import numpy as np
import pytest

from donof_b200 import Param, gnof, integrals, workload
from oracle import native
from test_digit_arithmetic import F, digits, product, truncated

ROW_SPREAD = 64.0
CASES = [("rows", "own"), ("rows", "near"), ("rows", "dense"), ("blocks", "own"),
         ("blocks", "dense"), ("mild", "own"), ("mild", "dense"), ("mild", "scaled"), ("molecule", "own"),
         ("molecule", "dense")]


def bounds(p, b, C, n, cj, ck):
    """Of b_pq[l, q, p], elag[a, b], J and K, from the largest elements of b's rows and C5's columns."""
    bl, C5 = np.abs(b).transpose(2, 0, 1), np.abs(C[:, :p.nbf5])
    dtmp = len(C) * 2.0 ** -44 * bl.max(2)[:, :, None] * C5.max(0)
    tmp = bl @ C5
    B = 2.0 * np.einsum("lmq,mp->lqp", dtmp, C5)
    bpq = np.einsum("lmq,mp->lqp", tmp, C5)
    at = np.arange(p.nbf5)

    def weights(x):                       # |W[l, q, b]| of |b_pq|
        w, t = np.abs(ck).T * x, x[:, at, at] * np.abs(n) + x[:, at, at] @ np.abs(cj).T
        w[:, at, at] += t
        return w

    Y = np.einsum("lmq,lqb->mb", dtmp, weights(bpq)) + np.einsum("lmq,lqb->mb", tmp, weights(B))
    dd, dB = bpq[:, at, at], B[:, at, at]
    J = np.einsum("lp,lq->pq", dd, dB)
    return B, 2.0 * np.abs(C).T @ Y, J + J.T, np.einsum("lqp,lqp->pq", 2.0 * bpq + B, B)


def system(kind, orbitals, seed=3):
    rng = np.random.default_rng(seed)
    if kind == "rows":
        nbf, naux = 48, 20
        b = workload.make_b(nbf, naux, rng).copy(order="F")
        for m, f in ((5, 1e-9), (9, 1e6), (11, 0.0)):
            b[m] *= f
            b[:, m] *= f
        S = np.eye(nbf)
    elif kind == "mild":                  # within what the digit products take
        nbf, naux = 48, 20
        g = 60.0 ** -rng.random(nbf)
        b = workload.make_b(nbf, naux, rng) * (g[:, None] * g)[:, :, None] / g.min()
        b = np.asfortranarray(b / np.sqrt(g.max()))
        S = np.eye(nbf)
    elif kind == "blocks":                # two fragments and the auxiliary functions of either
        nbf, naux = 40, 24
        b = np.zeros((nbf, nbf, naux), order="F")
        b[::2, ::2, :12] = workload.make_b(20, 12, rng)
        b[1::2, 1::2, 12:] = 1e-7 * workload.make_b(20, 12, rng)
        S = np.eye(nbf)
    else:                                 # two water molecules
        orb, aux = workload.water_cluster_bases(2, seed=seed)
        I, G = integrals.ERI_2e3c(orb, aux), integrals.ERI_2e2c(aux)
        w, V = np.linalg.eigh((G + G.T) / 2)
        b = np.asfortranarray(I.reshape(-1, len(w), order="F") @ ((V / np.sqrt(w)) @ V.T))
        nbf, naux = orb.nbas, aux.nbas
        b = b.reshape(nbf, nbf, naux, order="F")
        b = np.asfortranarray((b + b.transpose(1, 0, 2)) / 2)
        S = integrals.one_electron(orb)[0]
    p = Param(nbf=nbf, nbfaux=naux, nalpha=7, nbeta=7, ncwo=3)
    if orbitals == "own":                 # the basis functions themselves, orthogonalised
        s, U = np.linalg.eigh(S)
        C = (U / np.sqrt(s)) @ U.T
    elif orbitals == "near":
        C = np.linalg.qr(np.eye(nbf) + 1e-3 * rng.standard_normal((nbf, nbf)))[0]
    else:
        C = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0]
        if orbitals == "scaled":
            C *= 10.0 ** -rng.uniform(0, 9, nbf)
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    cj, ck = (np.asfortranarray(x) for x in gnof.coupling(n, p))
    return p, b, np.asfortranarray(C), n, cj, ck


def contract(p, b, C, n, cj, ck):
    """b_pq[l, q, p] and Y[m, b] as the kernels form them, and the spread of b's row norms."""
    bl, C5 = np.ascontiguousarray(b.transpose(2, 0, 1)), C[:, :p.nbf5]
    (db, sa), (dc, s1) = truncated(bl, 2), truncated(C5, 0)
    tmp = product(db, dc, 7, 7) * sa * s1
    norm = np.sqrt((bl * bl).sum(2))
    s = norm.max(1)[:, None, None] * np.sqrt((C5 * C5).sum(0)) * (1 + 2.0 ** -30) / F
    s[s == 0.0] = 1.0
    D, sb = digits(tmp, s), np.abs(C5).max(0) / F
    bpq = product([v.transpose(0, 2, 1) for v in D], digits(C5, sb), 8, 8) * s.transpose(0, 2, 1) * sb
    at, st = np.arange(p.nbf5), s.transpose(0, 2, 1)
    t = bpq[:, at, at] * np.where((at < p.nbeta) | (at >= p.nalpha), n, 0.0) + bpq[:, at, at] @ cj.T
    W = -ck.T * bpq
    W[:, at, at] += t
    beta = np.maximum(np.maximum(np.abs(ck).max(1), np.abs(cj).max(1)), np.abs(n))
    sw = (beta * np.abs(bpq * st).max((0, 1)) + np.abs(t * st[:, :, 0]).max(0)) / F
    sw[sw == 0.0] = 1.0
    Y = product([v.transpose(1, 0, 2).reshape(p.nbf, -1) for v in D],
                [v.reshape(-1, p.nbf5) for v in digits(W * st, sw)], 8, 8) * sw
    rows = norm.max(0)
    return bpq, Y, rows.max() / rows[rows > 0].min()


@pytest.mark.parametrize("kind,orbitals", CASES)
def test_the_scales_hold_every_element_to_its_bound(kind, orbitals):
    p, b, C, n, cj, ck = system(kind, orbitals)
    B, eb, jb, kb = bounds(p, b, C, n, cj, ck)
    bpq, Y, spread = contract(p, b, C, n, cj, ck)
    C5, H = C[:, :p.nbf5], np.zeros((p.nbf, p.nbf), order="F")
    e0, _ = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    held = (np.all(np.abs(bpq - np.einsum("mnl,np,mq->lqp", b, C5, C5, optimize=True)) <= B)
            and np.all(np.abs(C.T @ Y - e0[:, :p.nbf5]) <= eb))
    assert (spread > ROW_SPREAD) == (kind in ("rows", "blocks"))
    if spread <= ROW_SPREAD:
        J0, K0, _ = native.jkh_mo(C, H, b, p.nbf5)
        d = np.einsum("lpp->lp", bpq)
        assert held and np.all(np.abs(d.T @ d - J0) <= jb)
        assert np.all(np.abs((bpq * bpq).sum(0).T - K0) <= kb)
    elif (kind, orbitals) == ("rows", "own"):
        assert not held                    # the rule is needed
