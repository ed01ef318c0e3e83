"""The FP64 form's contractions from int8 digit slices (csrc/ozaki.cu) for an RI tensor
whose basis functions differ in size by many decades and for orbitals that do not mix
them, where every element has an error bound of its own (test_digit_scales.py derives
it); and T2 and Y for the tmp that T1 gave.
"""
import numpy as np
import pytest
import torch

import donof_b200 as d
from donof_b200 import Param, gnof, workload
from oracle import native
from test_digit_scales import CASES, bounds, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,orbitals", CASES)
def test_every_element_keeps_its_own_bound(cuda_ctx, kind, orbitals):
    p, b, C, n, cj, ck = system(kind, orbitals)
    H = np.zeros((p.nbf, p.nbf), order="F")  # elag is its two-electron part
    B, eb, jb, kb = bounds(p, b, C, n, cj, ck)
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    elag, _ = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    J, K, _ = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
    out = torch.empty((p.nbfaux, p.nbf5, p.nbf5), dtype=torch.float64, device="cuda")
    d.transform_dev(d.to_device(C), bt, p.nbf5, out=out)
    bpq = out.cpu().numpy()                # [l, q, p]
    bt.free()
    C5 = C[:, :p.nbf5]
    assert np.all(np.abs(bpq - np.einsum("mnl,np,mq->lqp", b, C5, C5, optimize=True)) <= B)
    e0, _ = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    J0, K0, _ = native.jkh_mo(C, H, b, p.nbf5)
    assert np.all(np.abs(J - J0) <= jb) and np.all(np.abs(K - K0) <= kb)
    assert np.all(np.abs(elag - e0)[:, :p.nbf5] <= eb)


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen", [(48, 20, 7, 3, 0), (129, 22, 16, 3, 1), (202, 37, 33, 5, 0),
                                                       (256, 30, 16, 3, 0), (300, 9, 20, 2, 0)])
def test_t2_and_y_are_as_near_as_fp64_products_of_the_same_tmp(cuda_ctx, nbf, naux, nbeta, ncwo, nopen):
    """b_pq and elag against FP64 products of the tmp that T1 gives.  tmp, C5 and W are
    rounded to 2^-57 of scales that lie 2^4 above their typical element, a relative error
    of 2^-53 of a term, and a sum of random terms has the relative error of its terms;
    the FP64 products on the other side err by sqrt(K) 2^-53 of theirs at most, K up to
    2^13 (elag of sums of 2^13 terms: 2^6.5 2^-53 = 1e-14 if nothing cancels; summed in
    blocks by BLAS, a tenth).  4e-15 leaves room for both, and is below what one digit
    of tmp less gives (restated on the CPU: b_pq 1.5e-14 and more, elag 4.4e-15 and more)."""
    rng = np.random.default_rng(nbf)
    p = Param(nbf=nbf, nbfaux=naux, nalpha=nbeta + nopen, nbeta=nbeta, ncwo=ncwo)
    b = workload.make_b(nbf, naux, rng)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    H = np.zeros((nbf, nbf), order="F")
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    cj, ck = (np.asfortranarray(x) for x in gnof.coupling(n, p))
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    tC = d.to_device(C)
    t1 = torch.empty((naux, p.nbf5, nbf), dtype=torch.float64, device="cuda")
    out = torch.empty((naux, p.nbf5, p.nbf5), dtype=torch.float64, device="cuda")
    d.t1_dev(tC, bt, p.nbf5, t1)
    d.transform_dev(tC, bt, p.nbf5, out=out)
    elag, _ = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    bt.free()
    tmp, bpq, C5 = t1.cpu().numpy(), out.cpu().numpy(), C[:, :p.nbf5]
    ref = tmp @ C5                         # [l, q, p]
    assert np.max(np.abs(bpq - ref)) <= 4e-15 * np.max(np.abs(ref))
    at = np.arange(p.nbf5)
    occ = np.where((at < p.nbeta) | (at >= p.nalpha), n, 0.0)
    W = -ck.T * ref                        # [l, q, b]
    W[:, at, at] += occ * ref[:, at, at] + ref[:, at, at] @ cj.T
    e0 = C.T @ np.einsum("lqm,lqb->mb", tmp, W, optimize=True)
    assert np.max(np.abs(elag[:, :p.nbf5] - e0)) <= 4e-15 * np.max(np.abs(e0))
