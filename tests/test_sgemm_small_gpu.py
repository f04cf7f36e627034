"""Small SGEMMs run on 8 x 16 tiles of 128 threads (64-k panels): the same bits as
the core's tiles, which compute every element as one FMA chain over k.  The
core's result comes from a product with more columns (too many tiles for the
small kernel, too little work for the tensor cores): edges of the tile, of the
panels, K = 1 and launches overlapping the call before."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (7, 15), (8, 16), (9, 17), (64, 64), (134, 76), (16, 1216), (152, 112)])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 63, 64, 65, 129, 200])
def test_same_bits_as_larger_tiles(dev, m, n, k):
    import torch
    from libgpublas_gb300._lib import _dp
    N = n + 16 * -(-100 // -(-m // 16))   # the larger product: at least 100 tiles of 16 x 16
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m * 7 + n + k)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float32, device="cuda", generator=gen) * 2 - 1
    a, b, c = uni(k, m), uni(N, k), uni(N, m)
    at, bt = a.T.contiguous(), b.T.contiguous()
    for ta, tb, alpha, beta in (("N", "N", 1.0, 1.0), ("T", "N", -0.5, 0.0), ("N", "T", 1.25, 0.75), ("T", "T", 1.0, 0.5)):
        x, ldx = (a, m) if ta == "N" else (at, k)
        y, ldy = (b, k) if tb == "N" else (bt, N)
        big, small = c.clone(), c[:n].clone()
        if beta == 0.0:
            small.fill_(float("nan"))
        torch.cuda.synchronize()
        for cols, out in ((N, big), (n, small)):
            assert dev.L.gbx_sgemm(dev.ctx, ta.encode(), tb.encode(), m, cols, k, alpha, _dp(x), ldx, _dp(y), ldy, beta,
                                   _dp(out), m) == 0
        dev.sync()
        assert torch.equal(small, big[:n])
