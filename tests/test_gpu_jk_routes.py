"""J_MO / K_MO partial sums (csrc/jk.cuh) on both sides of the lines between four (p, q)
per thread with staged diagonals and one with direct loads: nbf5 = 320 / 321 for FP32
b_pq (the mixed form), 512 / 513 for FP64.

Tolerances: those of test_gpu_w_and_jk_kernels.py."""
import pytest

import donof_b200 as d
from oracle import native

from test_gpu_digit_products import inputs, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol,nbf,naux,nbeta,ncwo,nopen", [
    ("mixed", 2e-4, 330, 11, 160, 1, 0), ("mixed", 2e-4, 330, 11, 160, 1, 1), ("mixed", 2e-4, 330, 1, 160, 1, 0),
    ("fp64", 1e-12, 516, 9, 256, 1, 0), ("fp64", 1e-12, 516, 9, 256, 1, 1)])
def test_jkh_mo(cuda_ctx, precision, tol, nbf, naux, nbeta, ncwo, nopen):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo, nopen, nbf)
    J0, K0, H0 = native.jkh_mo(C, H, b, p.nbf5)
    bt = d.eris_to_gpu(b, precision, cuda_ctx)
    J, K, Hc = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
    bt.free()
    assert rel(J, J0) <= tol and rel(K, K0) <= tol and rel(Hc, H0) <= 1e-12
