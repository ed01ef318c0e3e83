"""The FP64 form's contractions from int8 digit slices (csrc/ozaki.cu) at the sizes
where their tiles, chunks and paddings end, against the FP64 oracle.

Tolerance.  T1's operands carry 49 bits below a power of two at most twice the largest
element of the row (column), truncated, and the dropped digit products are of that size
too: for N(0, 1) b (elements up to 4) and orthonormal C the error of an element of tmp
is at most sqrt(nbf) 2^-46 from b's digits (sum_n |C| <= sqrt(nbf)) and as much from
C's.  tmp, W and T2's C5 carry 56 bits below bounds a few bits above their largest
element, and their dropped products lie below 2^-62 of the scales: less than the first.
Three contractions of nbf <= 400: 3 * 2 * 20 * 1.4e-14 < 4e-12 of the largest element.
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


def inputs(nbf, naux, nbeta, ncwo, nopen, seed=0):
    rng = np.random.default_rng(seed)
    p = Param(nbf=nbf, nbfaux=naux, nalpha=nbeta + nopen, nbeta=nbeta, ncwo=ncwo)
    b = workload.make_b(nbf, naux, rng)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    A = rng.standard_normal((nbf, nbf))
    H = np.asfortranarray((A + A.T) * (0.5 / np.sqrt(nbf)))
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    cj, ck = (np.asfortranarray(x) for x in gnof.coupling(n, p))
    return p, b, C, H, n, cj, ck


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen", [
    (1, 1, 1, 0, 0),         # a single element
    (17, 40, 5, 2, 0),       # nbf5 = 15: one padding column
    (32, 9, 4, 3, 0),        # nbf5 = 16
    (47, 31, 4, 3, 1),       # nbf5 = 17: a second group of 16
    (128, 21, 16, 3, 0),     # one K chunk, one column tile
    (129, 22, 16, 3, 1),     # two K chunks, nbf5 = 65: two column tiles
    (160, 150, 40, 3, 0),    # (q, l) over several chunks, K steps left out of the last n chunk
    (256, 3, 64, 3, 0),      # the last size with C5 resident; nbf5 = nbf
    (257, 7, 21, 2, 0),      # C5 streamed: three K chunks, nbf5 = 63
    (384, 5, 16, 2, 0),      # the last of them whole
    (385, 5, 16, 2, 2),      # a fourth
    (40, 2500, 10, 1, 0),    # a long (q, l) range: 625 chunks, more than one exact int32 range
])
def test_contractions_at_tile_edges_match_the_oracle(cuda_ctx, nbf, naux, nbeta, ncwo, nopen):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo, nopen, nbf + naux)
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    elag, Hmat, E = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta, return_energy=True)
    J, K, Hc = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
    bt.free()
    e0, h0 = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    J0, K0, H0 = native.jkh_mo(C, H, b, p.nbf5)
    assert rel(elag, e0) <= TOL and rel(Hmat, h0) <= TOL
    assert rel(J, J0) <= TOL and rel(K, K0) <= TOL and rel(Hc, H0) <= TOL


def test_a_context_with_fewer_ctas_than_column_tiles(cuda_ctx):
    """C5 cannot stay resident when a column tile has no CTA of its own: it streams, with the same sums."""
    p, b, C, H, n, cj, ck = inputs(200, 11, 33, 5, 0)
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    call = lambda: d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    whole = call()
    cuda_ctx.set_cta_limit(3)
    try:
        few = call()
    finally:
        cuda_ctx.set_cta_limit(0)
    bt.free()
    for x, y in zip(whole, few):
        assert rel(y, x) <= 1e-14


def test_zeros_and_non_finite_values(cuda_ctx):
    p, b, C, H, n, cj, ck = inputs(48, 20, 4, 3, 0)
    b = b.copy(order="F")
    b[:, :, 7] = 0.0                      # a zero b_l
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(True)
    C0 = C.copy(order="F")
    C0[:, 2] = 0.0                        # a zero orbital
    elag, _ = d.compute_Lagrange2(C0, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    assert rel(elag, native.lagrange2(C0, n, H, b, cj, ck, p.nalpha, p.nbeta)[0]) <= TOL
    z = np.zeros_like(cj)                 # every W is zero: Y = 0 and elag = C^T H C n
    elag, Hmat = d.compute_Lagrange2(C, n, H, bt, z, z, p.nalpha, 0)
    assert rel(elag[:, :p.nbf5], Hmat * n) <= 1e-14
    for bad in (np.nan, np.inf):          # no finite number stands where the FP64 GEMM gave none
        C1 = C.copy(order="F")
        C1[3, 1] = bad
        elag, _ = d.compute_Lagrange2(C1, n, H, bt, cj, ck, p.nalpha, p.nbeta)
        assert not np.any(np.isfinite(elag[:, :p.nbf5]))
    bt.free()
