"""The FP64 GEMM's narrow tiles (48 x 24 and 32 x 40, csrc/gemm_f64.cu) with rows and
columns just behind one of their tiles, at sizes that the tuner's rule admits them for.

The first call of a shape runs every candidate into the same output, the narrow ones last
(48 x 24, then 32 x 40), so the first call returns what the last admitted one wrote.  The
rule is restated here: a narrow tile is a candidate where it pads the result to less than
32 x 32 tiles do.

Tolerance: that of test_gpu_gemm_narrow_tiles.py."""
import numpy as np
import pytest

import donof_b200 as d
from oracle import native
from test_gpu_digit_products import inputs

pytestmark = pytest.mark.gpu
TOL = 1e-12


def candidates(M, N):
    pad = lambda m, n: -(-M // m) * m * (-(-N // n) * n)
    return [t for t in ((48, 24), (32, 40)) if pad(*t) < pad(32, 32)]


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen,last", [
    (97, 11, 8, 1, 1, (48, 24)),      # a row behind two tiles of 48; nbf5 = 17, part of a tile of 24
    (97, 9, 12, 1, 0, (48, 24)),      # ... nbf5 = 24, a whole one
    (96, 9, 10, 3, 1, (48, 24)),      # nbf5 = 41: a second tile of 24
    (33, 9, 16, 1, 1, (32, 40)),      # a row behind a tile of 32; nbf5 = 33, part of a tile of 40
    (65, 9, 20, 1, 0, (32, 40)),      # ... nbf5 = 40, a whole one
    (96, 9, 11, 5, 0, (32, 40)),      # nbf5 = 66: a second tile of 40, pairs of 16-byte copies
    (97, 7, 13, 5, 1, (32, 40)),      # nbf5 = 79, 8-byte copies
    (130, 5, 24, 3, 1, (32, 40)),     # nbf5 = 97: part of a third tile of 40, two rows behind tiles of 32
])
def test_behind_a_tile(cuda_ctx, nbf, naux, nbeta, ncwo, nopen, last):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo, nopen, nbf * naux)
    assert candidates(nbf, p.nbf5)[-1:] == [last]
    bt = d.eris_to_gpu(b, "fp64", cuda_ctx)
    bt.set_fp64_tc(False)
    e0, h0 = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    J0, K0, _ = native.jkh_mo(C, H, b, p.nbf5)
    for _ in range(2):
        elag, Hmat = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
        J, K, _ = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
        for x, x0 in ((elag, e0), (Hmat, h0), (J, J0), (K, K0)):
            assert np.max(np.abs(x - x0)) <= TOL * np.max(np.abs(x0))
    bt.free()
