"""donof_iaux takes the three-centre integrals from wherever one copy can: ordinary,
page-locked and device memory (above the size from which ordinary memory goes through
several host threads)."""
import ctypes as ct

import numpy as np
import pytest
import torch

import donof_b200 as d
from donof_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ordinary", "page-locked", "device"])
def test_where_the_integrals_lie(cuda_ctx, kind):
    nbf, n = 220, 64                       # 25 MB
    w = np.linspace(0.5, 4.0, n)
    G = np.asfortranarray(np.diag(w))
    I = torch.from_numpy(np.random.default_rng(0).standard_normal((n, nbf, nbf)))  # [l, n, m]
    src = {"ordinary": lambda: I, "page-locked": I.pin_memory, "device": I.cuda}[kind]()
    torch.cuda.synchronize()
    h = ct.c_void_p()
    cuda_ctx.check(cuda_ctx.lib.donof_iaux(cuda_ctx.handle, ct.c_void_p(G.ctypes.data), ct.c_void_p(src.data_ptr()), nbf,
                                           n, 0, ct.byref(h)))
    b = api.BTensor(cuda_ctx, h, nbf, n, 0)
    out = torch.zeros((n, nbf, nbf), dtype=torch.float64, device="cuda")
    d.transform_dev(d.to_device(np.asfortranarray(np.eye(nbf))), b, nbf, out=out)  # b itself
    torch.cuda.synchronize()
    b.free()
    ref = I.numpy() / np.sqrt(w)[:, None, None]
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1e-14 * np.max(np.abs(ref))  # G is diagonal: no rotation
