"""The in-place leaves of DTRSM: 64 x 64 inverted diagonal blocks times groups of
four or eight vectors.  Orders around 32, 64 and 128, vector counts around the
groups and around the count at which the groups grow (four vectors per SM); the
other triangle, a unit diagonal and the rows beyond m are NaN and stay so.

Tolerance: the triangle has a diagonal in [1, 2] and off-diagonal row and column
sums of at most 1/2, so |A| <= 2.5 and |inv| <= 2 in the infinity norm for either
side.  Inverting a block, multiplying by it and the products of the recursion
leave |B - op(A) X| <= 4 (na + 130) u |A| |inv| |A| |X|: 50 (na + 130) u max|X|."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na", [1, 31, 33, 63, 64, 65, 97, 129, 200])
@pytest.mark.parametrize("nvec", [1, 3, 4, 5, 9, 608, 609])
def test_solve(dev, na, nvec):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 * na + nvec)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    nan = float("nan")
    for side in "LR":
        m, n = (na, nvec) if side == "L" else (nvec, na)
        for uplo in "LU":
            for trans in "NT":
                for diag in "NU":
                    # tensors hold the transpose of the column-major matrix
                    off = uni(na, na) / (2 * na)
                    off = torch.triu(off, 1) if uplo == "L" else torch.tril(off, -1)
                    d = torch.ones(na, dtype=torch.float64, device="cuda") if diag == "U" else 1.5 + uni(na) / 2
                    a = (off + torch.diag(d)).T.contiguous()    # the matrix itself
                    keep = torch.tril(torch.ones_like(a), -1 if diag == "U" else 0) if uplo == "L" else \
                        torch.triu(torch.ones_like(a), 1 if diag == "U" else 0)
                    store = torch.full((na, na + 3), nan, dtype=torch.float64, device="cuda")
                    store[:, :na] = torch.where(keep.bool(), a, nan).T
                    b = torch.full((n, m + 5), nan, dtype=torch.float64, device="cuda")
                    b[:, :m] = uni(n, m)
                    x = b.clone()
                    torch.cuda.synchronize()
                    dev.dtrsm(side, uplo, trans, diag, m, n, -0.5, store, na + 3, x, m + 5)
                    dev.sync()
                    assert bool(torch.isnan(x[:, m:]).all())
                    op = a.T if trans == "T" else a
                    sol = x[:, :m].T
                    back = op @ sol if side == "L" else sol @ op
                    err = float((back - -0.5 * b[:, :m].T).abs().max())
                    assert err <= 50 * (na + 130) * 2.0 ** -53 * float(sol.abs().max())
