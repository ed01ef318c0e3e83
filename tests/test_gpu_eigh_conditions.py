"""The block Jacobi eigensolver (csrc/eigh.cu) on metrics like those of fitting sets:
eigenvalues over many decades, matrices of less than full rank (whose sweeps end when
the noise of the zero eigenvalues does), a molecule's own Coulomb metric, and with fewer
CTAs than block pairs.

Tolerance.  Rounding G moves its eigenvalues by up to n 2^-53 of the largest, w_max; that
is dw / (2 w) of the inverse square root along an eigenvector, and the smallest w makes
the largest element: n 2^-54 w_max / w_min of the norm of G^{-1/2}.
"""
import numpy as np
import pytest
import torch

import donof_b200 as d
from donof_b200 import _lib, integrals, workload

pytestmark = pytest.mark.gpu


def build(ctx, G, I):
    """b = I G^{-1/2}"""
    nbf, _, n = I.shape
    bt = d.Iaux_gpu(np.asfortranarray(G), np.asfortranarray(I), "fp64", ctx)
    out = torch.zeros(nbf * nbf * n, dtype=torch.float64, device="cuda")
    d.transform_dev(d.to_device(np.asfortranarray(np.eye(nbf))), bt, nbf, out=out)  # b itself
    torch.cuda.synchronize()
    bt.free()
    return out.cpu().numpy().reshape(nbf, nbf, n, order="F")


def symmetric(A):
    return np.triu(A) + np.triu(A, 1).T


@pytest.mark.parametrize("n", [96, 130])
@pytest.mark.parametrize("decades", [3, 6, 9, 12])
def test_eigenvalues_over_many_decades(cuda_ctx, n, decades):
    rng = np.random.default_rng(n + decades)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    w = np.logspace(-decades, 0, n)
    I = rng.standard_normal((4, 4, n))
    ref = I @ ((Q / np.sqrt(w)) @ Q.T)
    b = build(cuda_ctx, symmetric((Q * w) @ Q.T), I)
    assert np.max(np.abs(b - ref)) <= n * 2.0 ** -54 * 10.0 ** decades * np.max(np.abs(ref))


def test_a_coulomb_metric(cuda_ctx):
    aux = workload.water_cluster_bases(3, seed=1)[1]
    G = integrals.ERI_2e2c(aux)
    G = symmetric(G)
    n = len(G)
    I = np.random.default_rng(0).standard_normal((4, 4, n))
    w, V = np.linalg.eigh(G)
    ref = I @ ((V / np.sqrt(w)) @ V.T)
    assert np.max(np.abs(build(cuda_ctx, G, I) - ref)) <= 2 * n * 2.0 ** -54 * w[-1] / w[0] * np.max(np.abs(ref))


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("half rank", "repeated functions", "near zero")
                                    for n in (96, 320, 512)] + [("eighteen decades", 1024)])
def test_less_than_full_rank_ends(cuda_ctx, kind, n):
    """The sweeps end within their limit (rounding may leave an eigenvalue of exactly
    zero, whose b is refused as not finite).  In the space of the large eigenvalues b is
    theirs, but for what the computed eigenvectors of the others leak into it: an angle
    of n 2^-50 at most (w_max / w_min of the large ones is 8) times b's own size."""
    rng = np.random.default_rng(n)
    if kind == "half rank":
        B = np.linalg.qr(rng.standard_normal((n, n)))[0][:, :n // 2] * np.sqrt(np.linspace(0.5, 4.0, n // 2))
    elif kind == "repeated functions":     # a quarter of the functions stands in the set twice
        m = n - n // 4
        B = np.linalg.qr(rng.standard_normal((m, m)))[0] * np.sqrt(np.linspace(0.5, 4.0, m))
        B = B[np.r_[np.arange(m), np.arange(n - m)]]
    else:
        B = None
    if B is not None:
        G = symmetric(B @ B.T)
    else:
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        w = np.linspace(0.5, 4.0, n)
        w[:n // 8] = np.linspace(-1e-13, 1e-13, n // 8)
        if kind == "eighteen decades":
            w = np.logspace(-18, 0, n)
        G = symmetric((Q * w) @ Q.T)
    I = rng.standard_normal((4, 4, n))
    try:
        b = build(cuda_ctx, G, I)
    except _lib.DonofError as e:
        assert e.status == _lib.ERR_ARG
        return
    w, V = np.linalg.eigh(G)
    L, w = V[:, w > 0.25], w[w > 0.25]
    assert np.max(np.abs(b @ L - I @ (L / np.sqrt(w)))) <= n * 2.0 ** -50 * np.sqrt(n) * np.max(np.abs(b))


@pytest.mark.parametrize("ctas", [1, 2])
def test_fewer_ctas_than_block_pairs(cuda_ctx, ctas):
    """A CTA then takes several block pairs and tiles, with the same arithmetic."""
    n = 256
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    G = symmetric((Q * np.logspace(-3, 0, n)) @ Q.T)
    I = rng.standard_normal((4, 4, n))
    whole = build(cuda_ctx, G, I)
    cuda_ctx.set_cta_limit(ctas)
    try:
        few = build(cuda_ctx, G, I)
    finally:
        cuda_ctx.set_cta_limit(0)
    np.testing.assert_array_equal(few, whole)
