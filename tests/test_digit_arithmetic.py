"""The digit arithmetic of csrc/ozaki.cu restated on the CPU with exact integers:
seven truncated 7-bit digits for T1, seven balanced 8-bit digits from one 64-bit
addition for T2 and Y, the digit products with i + j < 7 and i + j < 8, and the
bounds that the kernel relies on."""
import numpy as np
import pytest

F, S = 0.498, 7


def truncated(x, axis):
    """S digits of x (most significant first) below a power of two per row or column, and that power."""
    s = 2.0 ** np.frexp(np.abs(x).max(axis, keepdims=True))[1]
    y, d = x / s, []
    for _ in range(S):
        y = y * 128.0
        d.append(np.trunc(y).astype(np.int64))
        y = y - d[-1]
    assert all(np.all(np.abs(v) <= 127) for v in d)
    return d, s


def digits(x, s):
    """S digits (most significant first) of x / s, |x| <= F s."""
    X = np.rint(x / s * 2.0 ** (8 * S)).astype(np.int64)
    bias = sum(128 << (8 * i) for i in range(S))
    z = X + bias                                  # the bytes of z are the digits + 128
    assert np.all(z >= 0) and np.all(z < 1 << (8 * S))
    d = [((z >> (8 * (S - 1 - i))) & 255) - 128 for i in range(S)]
    assert all(np.all(np.abs(v) <= 128) for v in d)
    assert np.array_equal(sum(v << (8 * (S - 1 - i)) for i, v in enumerate(d)), X)
    return d


def product(A, B, ng, bits):
    acc = [0] * ng
    for i, a in enumerate(A):
        for j, b in enumerate(B):
            if i + j < ng:
                acc[i + j] = acc[i + j] + a @ b
    assert all(np.all(np.abs(v) < 1 << 31) for v in acc)
    v = acc[-1].astype(np.float64)
    for a in reversed(acc[:-1]):
        v = v * 2.0 ** -bits + a
    return v * 2.0 ** (-2 * bits)


@pytest.mark.parametrize("nbf,naux,nbf5,scale", [(24, 5, 20, 0.0), (61, 3, 17, 0.0), (61, 3, 17, 6.0)])
def test_the_three_contractions(nbf, naux, nbf5, scale):
    """Within the 4e-12 that the GPU test allows (rows of b over `scale` decades too);
    T2 and Y, of the tmp and the W that they are given, within 1e-14."""
    rng = np.random.default_rng(nbf + nbf5)
    g = 10.0 ** rng.uniform(-scale, 0, nbf)
    b = rng.standard_normal((naux, nbf, nbf)) * g[:, None] * g
    C = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0][:, :nbf5]
    ck = rng.random((nbf5, nbf5))
    close = lambda x, x0, tol: np.max(np.abs(x - x0)) <= tol * np.max(np.abs(x0))
    tmp0 = b @ C
    (db, sa), (dc, s1) = truncated(b, 2), truncated(C, 0)
    tmp = product(db, dc, 7, 7) * sa * s1
    assert close(tmp, tmp0, 4e-12)
    # tmp's scale bounds it (Cauchy-Schwarz), so its digits always fit
    s = np.sqrt((b * b).sum(2)).max(1)[:, None, None] * np.sqrt((C * C).sum(0)) * (1 + 2.0 ** -30) / F
    D, sb = digits(tmp, s), np.abs(C).max(0) / F
    bpq0 = np.einsum("lmq,mp->lqp", tmp0, C)
    bpq = product([v.transpose(0, 2, 1) for v in D], digits(C, sb), 8, 8) * s.transpose(0, 2, 1) * sb
    assert close(bpq, bpq0, 4e-12) and close(bpq, np.einsum("lmq,mp->lqp", tmp, C), 1e-14)
    W = -ck * bpq * s.transpose(0, 2, 1)
    beta = np.abs(ck).max(0)
    sw = beta * np.abs(bpq * s.transpose(0, 2, 1)).max() / F
    Y = product([v.transpose(1, 0, 2).reshape(nbf, -1) for v in D], [v.reshape(-1, nbf5) for v in digits(W, sw)],
                8, 8) * sw
    Y0 = np.einsum("lmq,lqb->mb", tmp0, -ck * bpq0)
    assert close(Y, Y0, 4e-12) and close(Y, np.einsum("lmq,lqb->mb", tmp, -ck * bpq), 1e-14)


def test_the_extremes_fit():
    x = np.array([F, -F, 0.0, 0.5 ** 49, -0.5 ** 49, 1 / 256, -1 / 256, 127.49 / 256])
    digits(x, 1.0)
    assert 7 * 128 * 128 * 146 * 128 < 1 << 31    # the longest K range of one accumulation
