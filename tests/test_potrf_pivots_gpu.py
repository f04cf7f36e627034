"""gbx_dpotrf_small: the first non-positive pivot at every kind of place in a 32-column
step (first and last columns, either side of the 16th and of the eighths), in
the first and later steps, with and without a panel below."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 40, 100])
@pytest.mark.parametrize("col", [1, 2, 8, 9, 10, 16, 17, 18, 24, 25, 31, 32, 33, 34, 49, 64, 65, 100])
@pytest.mark.parametrize("value", [-1.0, 0.0, float("nan")])
def test_first_bad_pivot(dev, n, col, value):
    import torch
    if col > n:
        pytest.skip("beyond the matrix")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + col)
    # A = L D L^T with small integers: the pivots are exactly D, so a zero is found as one
    low = torch.randint(-1, 2, (n, n), device="cuda", generator=gen).double().tril(-1)
    low += torch.eye(n, dtype=torch.float64, device="cuda")
    d = torch.ones(n, dtype=torch.float64, device="cuda")
    d[col - 1] = 0.0 if value != value else value
    a = (low * d) @ low.T
    if value != value:
        a[col - 1, col - 1] = value
    info = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dev.dpotrf_small(n, a, n, info)
    dev.sync()
    assert int(info) == col
    good = (low @ low.T).contiguous()   # and the next call is not affected
    torch.cuda.synchronize()
    dev.dpotrf_small(n, good, n, info)
    dev.sync()
    assert int(info) == 0
    assert torch.equal(good.T.tril(), low)
