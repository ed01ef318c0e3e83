"""The Lagrangian tail's barrier state is zeroed by the kernels that build W (csrc/tail.cu):
a Lagrangian after JKH_MO, which writes over the same scratch, and a repeated one give the
first one's bits in every form; and so does the tail on another number of CTAs (a sum
does not depend on the grid)."""
import numpy as np
import pytest

import donof_b200 as d
from donof_b200 import Param, gnof, workload

pytestmark = pytest.mark.gpu


def inputs(nbf, naux, nbeta, ncwo):
    rng = np.random.default_rng(nbf)
    p = Param(nbf=nbf, nbfaux=naux, nalpha=nbeta, nbeta=nbeta, ncwo=ncwo)
    b = workload.make_b(nbf, naux, rng)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nbf, nbf)))[0])
    A = rng.standard_normal((nbf, nbf))
    H = np.asfortranarray((A + A.T) * (0.5 / np.sqrt(nbf)))
    n, _ = gnof.occupations(rng.standard_normal(p.nv), p)
    cj, ck = (np.asfortranarray(x) for x in gnof.coupling(n, p))
    return p, b, C, H, n, cj, ck


@pytest.mark.parametrize("form,nbf,naux,nbeta,ncwo", [
    ("fp64", 1, 1, 1, 0), ("fp64", 24, 20, 5, 3), ("fp64", 91, 30, 11, 5),
    ("fp64", 300, 4, 130, 1),            # nbf5 = 260: W's two kernels
    ("tc", 40, 20, 10, 1), ("mixed", 48, 20, 4, 3), ("mixed", 80, 12, 18, 3),
])
def test_repeated_lagrangians_around_jkh_agree(cuda_ctx, form, nbf, naux, nbeta, ncwo):
    p, b, C, H, n, cj, ck = inputs(nbf, naux, nbeta, ncwo)
    bt = d.eris_to_gpu(b, "mixed" if form == "mixed" else "fp64", cuda_ctx)
    if form != "mixed":
        bt.set_fp64_tc(form == "tc")
    call = lambda: d.compute_Lagrange2(C, n, H, bt, cj, ck, p.nalpha, p.nbeta, return_energy=True)
    call()                               # the autotuner's runs
    first = call()
    d.JKH_MO(C, H, bt, p.nbf, p.nbf5, p.nbfaux)
    for _ in range(2):
        for x, y in zip(first, call()):
            assert np.array_equal(x, y)
    if form == "fp64":
        cuda_ctx.set_cta_limit(2)
        try:
            few = call()
        finally:
            cuda_ctx.set_cta_limit(0)
        for x, y in zip(first, few):
            assert np.array_equal(x, y)
    bt.free()
