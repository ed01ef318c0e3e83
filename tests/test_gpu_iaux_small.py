"""Metrics smaller than the eigensolver's 64 x 64 block (csrc/eigh.cu rotates the circle of
their own indices, odd sizes with one dummy), and three-centre integrals on both sides of
256 KB (csrc/iaux.cu copies the smaller ones on the call's own stream).

Tolerance: that of test_gpu_eigh_blocks.py (eigenvalues within [0.5, 4])."""
import numpy as np
import pytest
import torch

import donof_b200 as d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbf,n", [(4, 1), (4, 2), (4, 3), (4, 4), (4, 7), (4, 16), (4, 33), (4, 62), (4, 63),
                                   (32, 32), (32, 33), (64, 8), (64, 9)])
def test_inverse_square_root(cuda_ctx, nbf, n):
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    w = np.linspace(0.5, 4.0, n)
    G = (Q * w) @ Q.T
    I = rng.standard_normal((nbf, nbf, n))
    b = d.Iaux_gpu(np.asfortranarray((G + G.T) / 2), np.asfortranarray(I), "fp64", cuda_ctx)
    out = torch.zeros(nbf * nbf * n, dtype=torch.float64, device="cuda")
    d.transform_dev(d.to_device(np.asfortranarray(np.eye(nbf))), b, nbf, out=out)  # b itself
    torch.cuda.synchronize()
    b.free()
    ref = I @ ((Q / np.sqrt(w)) @ Q.T)
    assert np.max(np.abs(out.cpu().numpy().reshape(nbf, nbf, n, order="F") - ref)) <= 1e-12 * np.max(np.abs(ref))
