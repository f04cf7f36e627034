"""DTRSV in slices of 16 rows: orders around a slice, a block of 64, the block
from which the product with the newest block is folded (8), and the number of
slices of a full grid (38 blocks on 152 SMs).

Tolerance: every row is a sum of products rounded to 2^-53 and a multiplication
by an inverted block of condition below 4: 1e-14 (90 u) of |op(A)| |x| in the
Frobenius norm, in which the row sums of rounding errors add up as squares."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 55, 56, 57, 63, 64, 65, 120, 511, 512, 513, 577, 640, 2431, 2432,
                               2433, 2497, 5000])
@pytest.mark.parametrize("uplo", "UL")
@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("diag", "NU")
def test_slices(dev, n, uplo, trans, diag):
    import torch
    from libgpublas_gb300._lib import _dp
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    ld = n + 3
    a = (torch.rand(n, ld, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1) / n
    a.diagonal().copy_(torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) + 1)
    b = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    t = a[:, :n].T
    t = t.tril() if uplo == "L" else t.triu()
    if diag == "U":
        t = t.clone()
        t.diagonal().fill_(1.0)
    # what is not read: the other triangle, a unit diagonal, the rows beyond n
    keep = torch.zeros(n, ld, dtype=torch.bool, device="cuda")
    ones = torch.ones(n, n, dtype=torch.bool, device="cuda")
    off = 1 if diag == "U" else 0
    keep[:, :n] = (ones.tril(-off) if uplo == "L" else ones.triu(off)).T
    a = torch.where(keep, a, float("nan"))
    op = t if trans == "N" else t.T
    for inc in (1, -2):
        x = torch.full((n * abs(inc),), 7.0, dtype=torch.float64, device="cuda")
        x[::abs(inc)] = b if inc > 0 else b.flip(0)
        torch.cuda.synchronize()
        st = dev.L.gbx_dtrsv(dev.ctx, uplo.encode(), trans.encode(), diag.encode(), n, _dp(a), ld, _dp(x), inc)
        assert st == 0
        dev.sync()
        got = x[::abs(inc)] if inc > 0 else x[::abs(inc)].flip(0)
        assert float((op @ got - b).norm()) <= 1e-14 * float(op.norm()) * float(got.norm())
        if inc == -2:
            assert bool((x[1::2] == 7.0).all())
