"""Grouped DTRSMs of ill-conditioned and badly scaled triangles: substitution is
backward stable row by row, whatever the triangle.

Tolerance, per element: forward substitution with one rounding per product leaves
|alpha B - op(A) X| <= (na + 3) u (|op(A)| |X| + |alpha B|) (Higham, Accuracy and
Stability of Numerical Algorithms, theorem 8.5; the quotient's and alpha's
roundings are two of the units), and 2^-1074 per operation where results are
subnormal.  The residual is formed in extended precision."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def triangle(kind, n, rng):
    """Lower triangular."""
    if kind == "kahan":      # inverse of size (1 + c)^n / s^n, well-scaled columns
        s, c = 0.8, 0.6
        return (s ** np.arange(n))[:, None] * (np.tril(np.full((n, n), -c), -1) + np.eye(n))
    if kind == "growing":    # 2^(n - 2) in the inverse
        return np.tril(-np.ones((n, n)), -1) + np.eye(n)
    t = np.tril(rng.uniform(-1, 1, (n, n)))
    if kind == "graded":
        return t * (10.0 ** rng.uniform(-8, 8, n))[:, None]
    if kind == "subnormal":  # reciprocals of the diagonal overflow
        return np.diag(4e-310 * (1 + np.arange(n) % 3)) + np.diag(np.full(n - 1, 1e-310), -1)
    if kind == "large":      # reciprocals of the diagonal are subnormal
        return np.tril(t, -1) * 1e305 + np.diag(np.full(n, 1.5e308))
    d = np.arange(n)         # "small pivots"
    t[d, d] = np.where(d % 3 == 1, 1e-9, 1.0)
    return t


@pytest.mark.parametrize("kind", ["kahan", "growing", "graded", "subnormal", "large", "small pivots"])
@pytest.mark.parametrize("side", "LR")
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("trans", "NT")
def test_backward_error(dev, kind, side, uplo, trans):
    import torch
    import libgpublas_gb300 as g
    rng = np.random.default_rng(5)
    ops, keep = [], []
    for na, nvec in itertools.product([5, 16, 17, 33, 40, 64, 100], [3, 16]):
        t = triangle(kind, na, rng)
        if uplo == "U":
            t = t[::-1, ::-1]
        a = t.T if trans == "T" else t   # op(A) = t: stored the other way round for T
        lower = (uplo == "L") != (trans == "T")
        x0 = rng.uniform(0.25, 0.5, (na, nvec))
        b = t @ x0 if side == "L" else x0.T @ t
        m, n = b.shape
        da = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
        dx = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
        keep.append((t, b, da, dx))
        ops.append(g.GbxOp(kind=2, side=side.encode(), uplo=b"L" if lower else b"U", transa=trans.encode(), diag=b"N",
                           m=m, n=n, alpha=1.0, A=da.data_ptr(), lda=na, C=dx.data_ptr(), ldc=m))
    torch.cuda.synchronize()
    plan = dev.plan_create(ops)
    dev.plan_launch(plan)
    dev.sync()
    dev.plan_destroy(plan)
    L = np.longdouble
    for t, b, _, dx in keep:
        x = dx.cpu().numpy().T
        na = len(t)
        assert np.isfinite(x).all()
        tl, xl, bl = t.astype(L), x.astype(L), b.astype(L)
        r = bl - (tl @ xl if side == "L" else xl @ tl)
        mag = np.abs(tl) @ np.abs(xl) if side == "L" else np.abs(xl) @ np.abs(tl)
        tol = (na + 3) * U * (mag + np.abs(bl)) + na * 2.0 ** -1074
        assert (np.abs(r) <= tol).all(), (na, float((np.abs(r) / tol).max()))


def test_special_values(dev):
    """A zero pivot gives an infinity or NaN, as division does; a zero's quotient keeps
    its sign."""
    import torch
    import libgpublas_gb300 as g
    n = 20
    t = np.diag(np.where(np.arange(n) % 2 == 0, 2.0, -3.0))
    t[7, 7] = 0.0
    b = np.zeros((n, 4))
    b[:, 1] = -0.0
    b[:, 2] = 1.0
    b[:, 3] = np.where(np.arange(n) == 3, np.inf, 6e-320)
    with np.errstate(all="ignore"):
        want = b / np.diag(t)[:, None]
    da, dx = torch.from_numpy(t.copy()).cuda(), torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    # the rows below row 3 of the last column subtract 0 * inf
    want[4:, 3] = np.nan
    want[8:, :2] = np.nan   # and those below the zero pivot 0 * NaN
    want[8:, 2] = np.nan    # 0 * inf
    torch.cuda.synchronize()
    plan = dev.plan_create([g.GbxOp(kind=2, side=b"L", uplo=b"L", transa=b"N", diag=b"N", m=n, n=4, alpha=1.0,
                                    A=da.data_ptr(), lda=n, C=dx.data_ptr(), ldc=n)])
    dev.plan_launch(plan)
    dev.sync()
    dev.plan_destroy(plan)
    got = dx.cpu().numpy().T
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(np.signbit(got[0]), np.signbit(want[0]))
