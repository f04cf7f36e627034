"""DTRSV of triangles whose diagonal blocks are ill-conditioned and whose other
blocks are large beside them: the solve must not lose more than the products with
the diagonal blocks' inverses do.

Tolerance, per element: forming the right-hand side of block s, a sum of n rounded
products, leaves 6 sqrt(n) u (|T| |x| + |b|), and its product with the inverse I of
the diagonal block D, whose own error is of the same form, 6 sqrt(2 64 + 16) u |D|
|I| (|D| |x|) (section 14.2 of Higham, Accuracy and Stability of Numerical
Algorithms, with the constants of a probabilistic analysis, Higham and Mary, SIAM J.
Sci. Comput. 41(5), 2019).  Nothing may be multiplied by the inverse that is
larger than |D| |x|: M = I T(s, s-1) formed beforehand would leave u |D| |I|
|T(s, s-1)| |x|.  Extended precision throughout."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U, NB = 2.0 ** -53, 64


def kahan(n, c, scale, rng):
    s = np.sqrt(1 - c * c)
    i = np.arange(n)
    t = (s ** (i % NB))[:, None] * (np.tril(np.full((n, n), -c), -1) + np.eye(n))
    for k in range(NB, n, NB):
        t[k:k + NB, :k] *= scale * rng.uniform(0.5, 1)
    return t


def plain(n, scale, rng):
    t = np.tril(rng.uniform(-1, 1, (n, n))) / n * scale
    np.fill_diagonal(t, rng.uniform(1, 2, n))
    return t


@pytest.mark.parametrize("uplo,trans", ["LN", "LT", "UN", "UT"])
@pytest.mark.parametrize("n", [640, 700, 1300, 2600])
@pytest.mark.parametrize("kind", ["kahan", "kahan, large blocks", "plain", "one bad block"])
def test_backward_error(dev, uplo, trans, n, kind):
    import torch
    rng = np.random.default_rng(n)
    if kind == "plain":
        t = plain(n, 1.0, rng)
    elif kind == "one bad block":   # the others are folded
        t = plain(n, 1.0, rng)
        k = slice(9 * NB, 10 * NB)
        m = len(range(n)[k])
        t[k, k] = kahan(m, 0.35, 1.0, rng)
        t[k, :9 * NB] *= 1e6
    else:
        t = kahan(n, 0.24, 1.0 if kind == "kahan" else 100.0, rng)   # (the error grows by it from block to block)
    x0 = rng.uniform(0.5, 1, n) * rng.choice([-1.0, 1.0], n)
    b = t @ x0
    # op(A) is t or, solved from the other end, t reversed
    op = t if (uplo == "L") == (trans == "N") else t[::-1, ::-1]
    rhs = b if (uplo == "L") == (trans == "N") else b[::-1]
    a = op if trans == "N" else op.T
    da = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    dx = torch.from_numpy(np.ascontiguousarray(rhs)).cuda()
    torch.cuda.synchronize()
    assert dev.L.gbx_dtrsv(dev.ctx, uplo.encode(), trans.encode(), b"N", n, C.c_void_p(da.data_ptr()), n,
                           C.c_void_p(dx.data_ptr()), 1) == 0
    dev.sync()
    x = dx.cpu().numpy()
    if (uplo == "L") != (trans == "N"):
        x = x[::-1]
    L = np.longdouble
    res = np.abs(b.astype(L) - (t.astype(L) * x.astype(L)).sum(1))
    mag = np.abs(t) @ np.abs(x) + np.abs(b)
    tol = 6 * n ** 0.5 * U * mag
    for k in range(0, n, NB):
        d = t[k:k + NB, k:k + NB].astype(L)
        inv = np.zeros_like(d)
        for i in range(len(d)):
            inv[i] = ((np.arange(len(d)) == i) - d[i, :i] @ inv[:i]) / d[i, i]
        tol[k:k + NB] += 6 * (2 * NB + 16) ** 0.5 * U * (np.abs(d) @ (np.abs(inv) @ (np.abs(d) @ np.abs(x[k:k + NB])))).astype(float)
    assert (res <= tol).all(), float((res / tol).max())
