"""Small FP64 products run on 8 x 16 tiles of 128 threads (64-k panels): the
same bits as the tile the core takes for a larger C, which computes every
element as one FMA chain over k.  Edges of the tile, of the panels and of the
skipped zero padding; K = 0 and 1; launches overlapping the call before."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (7, 15), (8, 16), (9, 17), (64, 64), (100, 120), (16, 1216), (152, 128)])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 63, 64, 65, 127, 129, 200])
def test_same_bits_as_larger_tiles(dev, m, n, k):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m * 7 + n + k)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    N = n + 3000   # the larger product: more columns, so a full grid of other tiles
    a, b, c = uni(k, m), uni(N, k), uni(N, m)
    at, bt = a.T.contiguous(), b.T.contiguous()
    for ta, tb, alpha, beta in (("N", "N", 1.0, 1.0), ("T", "N", -0.5, 0.0), ("N", "T", 1.25, 0.75)):
        x, ldx = (a, m) if ta == "N" else (at, k)
        y, ldy = (b, k) if tb == "N" else (bt, N)
        big, small = c.clone(), c[:n].clone()
        if beta == 0.0:
            small.fill_(float("nan"))
        torch.cuda.synchronize()
        assert dev.dgemm(ta, tb, m, N, k, alpha, x, ldx, y, ldy, beta, big, m) == 0
        assert dev.dgemm(ta, tb, m, n, k, alpha, x, ldx, y, ldy, beta, small, m) == 0
        dev.sync()
        assert torch.equal(small, big[:n])


def test_chain_of_dependent_calls(dev):
    """Each product reads the one before: C_(i+1) = C_i A, 40 calls in a row."""
    import torch
    n = 40
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    a = torch.linalg.qr(torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen))[0].contiguous()
    c = [torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) for _ in range(41)]
    torch.cuda.synchronize()
    for i in range(40):
        assert dev.dgemm("N", "N", n, n, n, 1.0, c[i], n, a, n, 0.0, c[i + 1], n) == 0
    dev.sync()
    # column-major: C_(i+1)^T = A^T C_i^T on the tensors
    ref = c[0]
    for _ in range(40):
        ref = a @ ref
    assert float((c[40] - ref).norm()) <= 40 * n * 2.0 ** -53 * float(ref.norm())
