"""The digit arithmetic of csrc/ozaki.cu restated on the CPU with exact integers:
balanced 8-bit digits from one 64-bit addition, 6 digits of b and C5, 7 of tmp and
W, the digit products with i + j < 7, and the bounds that the kernel relies on."""
import numpy as np
import pytest

F, NG = 0.498, 7


def digits(x, s, count):
    """count digits (most significant first) of x / s, |x| <= F s."""
    X = np.rint(x / s * 2.0 ** (8 * count)).astype(np.int64)
    bias = sum(128 << (8 * i) for i in range(count))
    z = X + bias                                  # the bytes of z are the digits + 128
    assert np.all(z >= 0) and np.all(z < 1 << (8 * count))
    d = [((z >> (8 * (count - 1 - i))) & 255) - 128 for i in range(count)]
    assert all(np.all(np.abs(v) <= 128) for v in d)
    assert np.array_equal(sum(v << (8 * (count - 1 - i)) for i, v in enumerate(d)), X)
    return d


def product(A, B):
    acc = [0] * NG
    for i, a in enumerate(A):
        for j, b in enumerate(B):
            if i + j < NG:
                acc[i + j] = acc[i + j] + a @ b
    assert all(np.all(np.abs(v) < 1 << 31) for v in acc)
    v = acc[-1].astype(np.float64)
    for a in reversed(acc[:-1]):
        v = v * 2.0 ** -8 + a
    return v * 2.0 ** -16


@pytest.mark.parametrize("nbf,naux,nbf5,scale", [(24, 5, 20, 0.0), (61, 3, 17, 0.0), (61, 3, 17, 6.0)])
def test_the_three_contractions(nbf, naux, nbf5, scale):
    """Within the 4e-12 that the GPU test allows (rows of b over `scale` decades too)."""
    rng = np.random.default_rng(nbf + nbf5)
    g = 10.0 ** rng.uniform(-scale, 0, nbf)
    b = rng.standard_normal((naux, nbf, nbf)) * g[:, None] * g
    C = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0][:, :nbf5]
    ck = rng.random((nbf5, nbf5))
    tmp0 = b @ C
    sa, sb = np.abs(b).max(2, keepdims=True) / F, np.abs(C).max(0) / F
    tmp = product(digits(b, sa, 6), digits(C, sb, 6)) * sa * sb
    assert np.max(np.abs(tmp - tmp0)) <= 4e-12 * np.max(np.abs(tmp0))
    # tmp's scale bounds it (Cauchy-Schwarz), so its digits always fit
    s = np.sqrt((b * b).sum(2)).max(1)[:, None, None] * np.sqrt((C * C).sum(0)) * (1 + 2.0 ** -30) / F
    D = digits(tmp, s, 7)
    bpq0 = np.einsum("lmq,mp->lqp", tmp0, C)
    bpq = product([v.transpose(0, 2, 1) for v in D], digits(C, sb, 6)) * s.transpose(0, 2, 1) * sb
    assert np.max(np.abs(bpq - bpq0)) <= 4e-12 * np.max(np.abs(bpq0))
    W = -ck * bpq * s.transpose(0, 2, 1)
    beta = np.abs(ck).max(0)
    sw = beta * np.abs(bpq * s.transpose(0, 2, 1)).max() / F
    Y = product([v.transpose(1, 0, 2).reshape(nbf, -1) for v in D], [v.reshape(-1, nbf5) for v in digits(W, sw, 7)]) * sw
    Y0 = np.einsum("lmq,lqb->mb", tmp0, -ck * bpq0)
    assert np.max(np.abs(Y - Y0)) <= 4e-12 * np.max(np.abs(Y0))


def test_the_extremes_fit():
    x = np.array([F, -F, 0.0, 0.5 ** 49, -0.5 ** 49, 1 / 256, -1 / 256, 127.49 / 256])
    for count in (6, 7):
        digits(x, 1.0, count)
    assert 7 * 128 * 128 * 146 * 128 < 1 << 31    # the longest K range of one accumulation
