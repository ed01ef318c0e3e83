"""J_MO / K_MO partial sums (csrc/jk.cuh) and the general mixed form's W kernels
(csrc/mixed_general.cu) where their paths change: one or four (p, q) per thread
(nbf5 90 / 91), rows of W over one or two passes of 256 q (nbf5 257), diagonals in
one panel of 512 or two (nbf5 513), aux counts that leave a remainder of 8.

FP64 tolerance: sums of at most 2 nbf + naux products, each rounded at 1.1e-16:
(2 * 520 + 61) * 1.1e-16 < 2e-13 of the largest element if every rounding added up;
1e-12.  Mixed: the 2e-4 of the split representation (16 significant bits)."""
import numpy as np
import pytest

import donof_b200 as d
from oracle import native

from test_gpu_digit_products import inputs, rel

pytestmark = pytest.mark.gpu
SHAPES = [(96, 61, 15, 5, 0), (96, 61, 13, 6, 0), (130, 13, 16, 7, 0), (260, 9, 128, 1, 1), (520, 5, 171, 2, 0)]


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen", SHAPES)
def test_jkh_mo(cuda_ctx, nbf, naux, nbeta, ncwo, nopen):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo, nopen, nbf)
    J0, K0, H0 = native.jkh_mo(C, H, b, p.nbf5)
    for precision, tol in (("fp64", 1e-12), ("mixed", 2e-4)):
        bt = d.eris_to_gpu(b, precision, cuda_ctx)
        J, K, Hc = d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
        bt.free()
        assert rel(J, J0) <= tol and rel(K, K0) <= tol and rel(Hc, H0) <= 1e-12


@pytest.mark.parametrize("nbf,naux,nbeta,ncwo,nopen", SHAPES)
def test_mixed_lagrangian(cuda_ctx, nbf, naux, nbeta, ncwo, nopen):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo, nopen, nbf)
    bt = d.eris_to_gpu(b, "mixed", cuda_ctx)
    elag, Hmat = d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta)
    bt.free()
    e0, h0 = native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)
    assert rel(elag, e0) <= 2e-4 and rel(Hmat, h0) <= 1e-12


def test_grouped_products_with_fewer_ctas_than_tiles(cuda_ctx):
    """A context with a share of the SMs walks the grouped GEMMs' tile list: same tiles, same sums."""
    import torch

    cases = [inputs(24, 60, 5, 3, 0, 1), inputs(61, 40, 9, 4, 1, 2), inputs(96, 33, 20, 3, 0, 3)]
    jobs = [d.eris_to_gpu(c[1], "fp64", cuda_ctx) for c in cases]
    batch = d.Batch(jobs, [c[0] for c in cases], cuda_ctx)
    dev = [[d.to_device(x) for x in (c[4], c[5], c[6], c[3], c[2])] for c in cases]  # n, cj, ck, H, C

    def call():
        elag = [torch.zeros(c[0].nbf, c[0].nbf, dtype=torch.float64, device="cuda") for c in cases]
        hmat = [torch.zeros(c[0].nbf5, c[0].nbf, dtype=torch.float64, device="cuda") for c in cases]
        batch.lagrange2(*[[x[k] for x in dev] for k in range(5)], elag, hmat)
        torch.cuda.synchronize()
        return [d.from_device(x) for x in elag]

    whole = call()
    cuda_ctx.set_cta_limit(7)
    try:
        few = call()
    finally:
        cuda_ctx.set_cta_limit(0)
    batch.free()
    for (p, b, C, H, n, cj, ck), x, y in zip(cases, whole, few):
        assert rel(x, native.lagrange2(C, n, H, b, cj, ck, p.nalpha, p.nbeta)[0]) <= 1e-12
        assert rel(y, x) <= 1e-14
