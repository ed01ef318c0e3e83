"""The block Jacobi eigensolver (csrc/eigh.cu) at the edges of its 32-blocks and
64-wide pairs (one pair, odd and even numbers of pairs, one index more or less),
over scales that its angle's exponent arithmetic has to carry, and for a matrix
that needs no rotation.

Tolerance: eigenvalues within [0.5, 4] of each other, so G^{-1/2} has condition 3;
12 sweeps of n rotations per column leave about sqrt(12 n) 1.1e-16 per element,
5e-15 of the norm at n = 192, and the products with I a similar amount: 1e-12.
"""
import numpy as np
import pytest
import torch

import donof_b200 as d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,scale,kind", [
    (1, 1.0, "dense"), (2, 1.0, "dense"), (31, 1.0, "dense"), (63, 1.0, "dense"), (64, 1.0, "dense"),
    (65, 1.0, "dense"), (128, 1.0, "dense"), (129, 1.0, "dense"), (192, 1.0, "dense"),
    (70, 1e-100, "dense"), (70, 1e100, "dense"), (96, 1.0, "diagonal"), (96, 1.0, "two blocks"),
])
def test_inverse_square_root(cuda_ctx, n, scale, kind):
    rng = np.random.default_rng(n)
    w = np.linspace(0.5, 4.0, n)
    if kind == "dense":
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    elif kind == "diagonal":
        Q = np.eye(n)
    else:  # no coupling between the two halves
        Q = np.zeros((n, n))
        for s in (slice(0, n // 2), slice(n // 2, n)):
            Q[s, s] = np.linalg.qr(rng.standard_normal((n // 2, n // 2)))[0]
    G = np.asfortranarray((Q * (w * scale)) @ Q.T)
    I = np.asfortranarray(rng.standard_normal((4, 4, n)))
    b = d.Iaux_gpu(G, I, "fp64", cuda_ctx)
    out = torch.zeros(16 * n, dtype=torch.float64, device="cuda")
    d.transform_dev(d.to_device(np.asfortranarray(np.eye(4))), b, 4, out=out)  # b itself
    torch.cuda.synchronize()
    b.free()
    ref = I @ ((Q / np.sqrt(w * scale)) @ Q.T)
    got = out.cpu().numpy().reshape(4, 4, n, order="F")
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
