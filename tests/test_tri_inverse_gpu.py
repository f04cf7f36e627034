"""DTRSV, DTRSM and the DTRSM through the inverse, whose diagonal blocks are
inverted: triangles whose inverse, joined from those of smaller blocks, would have
lost the blocks' condition number once more (Cholesky factors of Gaussian kernels),
well-conditioned ones, and singular ones.

Tolerance: the same method restated in numpy, blocks inverted by substitution,
column by column, gives the backward error that the method has on these operands;
rounding errors that are of the same size and independent differ between two
orders of summation by small factors, of which 10 is allowed, plus 40 u for the
well-conditioned ones.  (The joined inverse: 30 to 4000.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U, NB = 2.0 ** -53, 64


def kernel(n, g, e):
    t = np.linspace(0, 1, n)
    return np.linalg.cholesky(np.exp(-(t[:, None] - t) ** 2 * g) + e * np.eye(n))


def inverse(d):
    x, s = np.zeros_like(d), np.eye(len(d))
    for i in range(len(d)):
        x[i] = s[i] / d[i, i]
        s[i + 1:] -= np.outer(d[i + 1:, i], x[i])
    return x


def solve(t, b):
    x = np.zeros_like(b)
    for k in range(0, len(t), NB):
        x[k:k + NB] = inverse(t[k:k + NB, k:k + NB]) @ (b[k:k + NB] - t[k:k + NB, :k] @ x[:k])
    return x


def backward(t, x, b):
    L = np.longdouble
    res = np.abs(b.astype(L) - t.astype(L) @ x.astype(L))
    return float((res / (np.abs(t) @ np.abs(x) + np.abs(b))).max())


KINDS = [(500, 1e-6), (500, 1e-8), (1000, 1e-10), (200, 1e-8), None]


def triangle(kind, n, rng):
    if kind:
        return kernel(n, kind[0] * n / 256, kind[1])   # neighbours as far apart as at n = 256 at most
    t = np.tril(rng.uniform(-1, 1, (n, n))) / n
    np.fill_diagonal(t, rng.uniform(1, 2, n))
    return t


def dev_matrix(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("uplo,trans", ["LN", "LT", "UN", "UT"])
@pytest.mark.parametrize("n", [50, 64, 130, 256])
@pytest.mark.parametrize("call", ["dtrsv", "dtrsm left", "dtrsm right", "dtrsm_ozaki left", "dtrsm_ozaki right"])
def test_backward_error(dev, kind, uplo, trans, n, call):
    import torch
    rng = np.random.default_rng(n)
    t = triangle(kind, n, rng)
    rhs = 1 if call == "dtrsv" else 5
    b = t @ (rng.uniform(0.5, 1, (n, rhs)) * rng.choice([-1.0, 1.0], (n, rhs)))
    right = call.endswith("right")
    # solves with op(A) = t, or from the other end with t reversed; on the right with its transpose
    forward = ((uplo == "L") == (trans == "N")) != right
    f = slice(None) if forward else slice(None, None, -1)
    op = t[f, f].T if right else t[f, f]
    da = dev_matrix(op if trans == "N" else op.T)
    dx = dev_matrix(b[f].T if right else b[f])
    torch.cuda.synchronize()
    if call == "dtrsv":
        assert dev.L.gbx_dtrsv(dev.ctx, uplo.encode(), trans.encode(), b"N", n, C.c_void_p(da.data_ptr()), n,
                               C.c_void_p(dx.data_ptr()), 1) == 0
    else:
        m, k, side = (rhs, n, "R") if right else (n, rhs, "L")
        if "ozaki" in call:
            dev.dtrsm_ozaki(side, uplo, trans, "N", m, k, 1.0, da, n, dx, m, slices=14)   # 70 bits
        else:
            dev.dtrsm(side, uplo, trans, "N", m, k, 1.0, da, n, dx, m)
    dev.sync()
    x = dx.cpu().numpy() if right else dx.cpu().numpy().T
    x = x[f]
    ref = inverse(t) @ b if "ozaki" in call else solve(t, b)
    assert backward(t, x, b) <= 10 * backward(t, ref, b) + 40 * U, (backward(t, x, b), backward(t, ref, b))


@pytest.mark.parametrize("call", ["dtrsv", "dtrsm", "dtrsm_ozaki"])
def test_zero_pivot(dev, call):
    """Rows before a zero pivot are solved as ever."""
    import torch
    n, z = 100, 70
    rng = np.random.default_rng(1)
    t = triangle(None, n, rng)
    t[z, z] = 0.0
    b = t @ rng.uniform(0.5, 1, (n, 1))
    da, dx = dev_matrix(t), dev_matrix(b)
    torch.cuda.synchronize()
    if call == "dtrsv":
        assert dev.L.gbx_dtrsv(dev.ctx, b"L", b"N", b"N", n, C.c_void_p(da.data_ptr()), n, C.c_void_p(dx.data_ptr()), 1) == 0
    elif call == "dtrsm":
        dev.dtrsm("L", "L", "N", "N", n, 1, 1.0, da, n, dx, n)
    else:
        assert dev.L.gbx_dtrsm_ozaki(dev.ctx, b"L", b"L", b"N", b"N", n, 1, C.c_double(1.0), C.c_void_p(da.data_ptr()), n,
                                     C.c_void_p(dx.data_ptr()), n, C.c_double(0.0), 0, None) == 0
    if call != "dtrsm_ozaki":
        dev.sync()
        x = dx.cpu().numpy().T
        k = z // NB * NB   # whole blocks before it
        assert backward(t[:k, :k], x[:k], b[:k]) <= 40 * U
        assert not np.isfinite(x[z]).any()
    else:
        assert dev.L.gbx_ctx_sync(dev.ctx) != 0   # the product reports its non-finite operand
