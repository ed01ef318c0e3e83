"""With b's digit slices on the device, T2 and Y run from digits or as FP64 GEMMs of T1's
tmp, by a rule on nbf and nbf5 (csrc/ozaki.cu).  Both sides of its line against the FP64
oracle, in one job that crosses it from call to call (the scratch is shared), with zeros
and values that are not finite.

Tolerance: T1's bound of test_gpu_digit_products.py, 4e-12 of the largest element.
"""
import numpy as np
import pytest

import donof_b200 as d
from donof_b200 import Param, gnof, workload
from oracle import native

pytestmark = pytest.mark.gpu
TOL = 4e-12


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def functional(p, rng):
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    return (n, *(np.asfortranarray(x) for x in gnof.coupling(n, p)))


def check(bt, b, C, H, p, rng):
    n, cj, ck = functional(p, rng)
    elag, Hmat = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    J, K, Hc = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
    e0, h0 = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    J0, K0, H0 = native.jkh_mo(C, H, b, p.nbf5)
    for x, x0 in ((elag, e0), (Hmat, h0), (J, J0), (K, K0), (Hc, H0)):
        assert rel(x, x0) <= TOL


@pytest.mark.parametrize("nbf,naux,functionals", [
    (128, 21, [(6, 3, 1), (6, 3, 0), (2, 1, 0), (6, 3, 1), (1, 0, 0)]),  # nbf5 = 25, 24, 4, 25, 1
    (223, 5, [(4, 3, 0), (6, 3, 1)]),
    (224, 5, [(4, 3, 0), (6, 3, 0), (1, 0, 0)]),                         # from digits whatever nbf5
    (33, 40, [(10, 2, 1)]),          # nbf5 = 31: one padding column
    (32, 9, [(8, 3, 0)]),            # nbf5 = 32: none
    (47, 31, [(8, 3, 1)]),           # nbf5 = 33: a third group of 16
    (40, 2500, [(6, 3, 1)]),         # a long (q, l) range: 625 chunks, more than one exact int32 range
])
def test_both_sides_of_the_line(cuda_ctx, nbf, naux, functionals):
    rng = np.random.default_rng(nbf)
    b = workload.make_b(nbf, naux, rng)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    H = rng.standard_normal((nbf, nbf))
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    for nbeta, ncwo, nopen in functionals:
        check(bt, b, C, np.asfortranarray(H + H.T),
              Param(nbf=nbf, nbfaux=naux, nalpha=nbeta + nopen, nbeta=nbeta, ncwo=ncwo), rng)
    bt.free()


@pytest.mark.parametrize("nopen", [0, 1])
def test_zeros_and_non_finite_values(cuda_ctx, nopen):
    rng = np.random.default_rng(48)
    nbf, naux = 48, 20
    p = Param(nbf=nbf, nbfaux=naux, nalpha=6 + nopen, nbeta=6, ncwo=3)  # nbf5 = 24 or 25
    n, cj, ck = functional(p, rng)
    b = workload.make_b(nbf, naux, rng).copy(order="F")
    b[:, :, 7] = 0.0
    b[5] = 0.0
    b[:, 5] = 0.0
    H = np.zeros((nbf, nbf), order="F")
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    C[:, 2] = 0.0
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    elag, _ = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    assert rel(elag, native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)[0]) <= TOL
    z = np.zeros_like(cj)
    elag, _ = d.compute_Lagrange2(C, n, H, bt, z, z, p.nalpha, 0)      # W = 0
    assert np.all(elag == 0.0)
    for bad in (np.nan, np.inf):          # in an orbital of C5: no finite number in the columns of elag
        C1 = C.copy(order="F")
        C1[3, 1] = bad
        elag, _ = d.compute_Lagrange2(C1, n, H, bt, cj, ck, p.nalpha, p.nbeta)
        assert not np.any(np.isfinite(elag[:, :p.nbf5]))
    n1 = n.copy()
    n1[1] = np.nan                        # of one orbital's weights: that column alone
    elag, _ = d.compute_Lagrange2(C, n1, H, bt, cj, ck, p.nalpha, p.nbeta)
    assert np.all(np.isnan(elag[:, 1])) and np.all(np.isfinite(np.delete(elag, 1, axis=1)))
    bt.free()
