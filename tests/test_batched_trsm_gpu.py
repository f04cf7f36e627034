"""Grouped DTRSMs solved in blocks of 16 rows: orders and system counts around the
blocks, every side, triangle, transposition and diagonal; the other triangle is
NaN.

Tolerance: the triangle has a diagonal in [1, 2] and off-diagonal row and column
sums of at most 1/2 (|A| <= 2.5, |inv| <= 2): inverting a block, multiplying by
it and the subtractions leave |B - op(A) X| <= 4 (na + 40) u |A| |inv| |A| |X|, so
50 (na + 40) u max|X|."""
import itertools

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", "LR")
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("diag", "NU")
def test_blocks(dev, side, uplo, trans, diag):
    import torch
    import libgpublas_gb300 as g
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    ops, keep = [], []
    for na, nvec in itertools.product([1, 2, 15, 16, 17, 31, 32, 33, 48, 100, 255, 256], [1, 15, 16, 17, 40]):
        m, n = (na, nvec) if side == "L" else (nvec, na)
        off = uni(na, na) / (2 * na)
        off = off.tril(-1) if uplo == "L" else off.triu(1)
        d = torch.ones(na, dtype=torch.float64, device="cuda") if diag == "U" else 1.5 + uni(na) / 2
        a = off + torch.diag(d)
        ones = torch.ones(na, na, dtype=torch.bool, device="cuda")
        k = 1 if diag == "U" else 0
        stored = ones.tril(-k) if uplo == "L" else ones.triu(k)
        store = torch.full((na, na + 1), float("nan"), dtype=torch.float64, device="cuda")
        store[:, :na] = torch.where(stored, a, float("nan")).T
        b = uni(n, m + 2)
        x = b.clone()
        keep.append((a, store, b, x, m, n, na))
        ops.append(g.GbxOp(kind=2, side=side.encode(), uplo=uplo.encode(), transa=trans.encode(), diag=diag.encode(), m=m,
                           n=n, alpha=-0.5, A=store.data_ptr(), lda=na + 1, C=x.data_ptr(), ldc=m + 2))
    torch.cuda.synchronize()
    plan = dev.plan_create(ops)
    dev.plan_launch(plan)
    dev.sync()
    dev.plan_destroy(plan)
    for a, store, b, x, m, n, na in keep:
        assert torch.equal(x[:, m:], b[:, m:])
        op = a.T if trans == "T" else a
        sol = x[:, :m].T
        back = op @ sol if side == "L" else sol @ op
        err = float((back + 0.5 * b[:, :m].T).abs().max())
        assert err <= 50 * (na + 40) * 2.0 ** -53 * float(sol.abs().max()), (na, m, n)
