"""The FP64 GEMM's narrow tiles (48 x 24 and 32 x 40, csrc/gemm_f64.cu) at the edges of
their tiles, against the FP64 oracle.

The first call of a shape runs every candidate into the same output, a narrow one last
where it pads the result less than 32 x 32 tiles do, so it is what the first call
returns; the second call runs the one that was chosen, with the same sums.

Tolerance.  Both sides are FP64 sums of n < 2^11 products (n = nbf, then nbf5 naux) in
different orders, over three contractions: sqrt(n) 2^-53 each in units of the terms'
size, 3 * 45 * 1.1e-16 = 1.5e-14, and the largest element of a result is not smaller
than its typical term: 1e-12 leaves a factor 60.
"""
import numpy as np
import pytest

import donof_b200 as d
from donof_b200 import Param, gnof, workload
from oracle import native

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen", [
    (40, 19, 10, 1, 0),      # nbf5 = 20: 48 x 24 is last for T1
    (48, 23, 8, 2, 0),       # nbf5 = 24: one whole tile
    (72, 17, 9, 3, 0),       # nbf5 = 36: one tile of 40
    (80, 21, 20, 1, 0),      # nbf5 = 40 = one whole tile of 40, pairs of 16-byte copies
    (91, 13, 11, 5, 0),      # odd: 8-byte copies; nbf5 = 66, three tiles of 24
    (67, 11, 12, 2, 1),      # nbf5 = 37
    (97, 31, 10, 3, 1),      # nbf5 = 41: a column behind a tile of 40
    (33, 9, 16, 1, 0),       # a row behind a tile of 32
])
def test_narrow_tiles_match_the_oracle(cuda_ctx, nbf, naux, nbeta, ncwo, nopen):
    rng = np.random.default_rng(nbf * naux)
    p = Param(nbf=nbf, nbfaux=naux, nalpha=nbeta + nopen, nbeta=nbeta, ncwo=ncwo)
    b = workload.make_b(nbf, naux, rng)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    A = rng.standard_normal((nbf, nbf))
    H = np.asfortranarray((A + A.T) * (0.5 / np.sqrt(nbf)))
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    cj, ck = (np.asfortranarray(x) for x in gnof.coupling(n, p))
    e0, h0 = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    J0, K0, _ = native.jkh_mo(C, H, b, p.nbf5)
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(False)
    for _ in range(2):
        elag, Hmat = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
        J, K, _ = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
        for x, x0 in ((elag, e0), (Hmat, h0), (J, J0), (K, K0)):
            assert np.max(np.abs(x - x0)) <= TOL * np.max(np.abs(x0))
    bt.free()
