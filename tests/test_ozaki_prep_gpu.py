"""The one-launch preparation of small-K Ozaki products (four rows per CTA,
four consecutive k per thread, passes of 256 k) at the edges of its blocks, for
operands in every storage order, entries over 2^-20 .. 2^20, and for both of
its launch forms (few and many blocks).  The error target of the call is 1e-14
relative (Frobenius); the 64-bit product it is compared with is within k 2^-53
of exact per entry, below 1e-14 of the norm at these sizes: 2e-14 in all."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 4), (4, 16, 127), (5, 17, 128), (127, 130, 129), (129, 33, 255),
                                   (64, 64, 256), (130, 70, 257), (33, 1, 513), (130, 257, 1023), (257, 19, 1024),
                                   (4100, 300, 256), (3000, 1300, 300)])
@pytest.mark.parametrize("ta,tb", ["NN", "TN", "NT", "TT"])
def test_small_k(dev, m, n, k, ta, tb):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n + k)

    def make(r, c):
        x = torch.rand(r, c, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        return torch.ldexp(x, torch.randint(-20, 21, (r, c), device="cuda", generator=gen))
    pad = m % 2
    a = make(*((k, m + pad) if ta == "N" else (m, k + pad)))
    b = make(*((n, k + pad) if tb == "N" else (k, n + pad)))
    opa = a[:, :m].T if ta == "N" else a[:, :k]
    opb = b[:, :k].T if tb == "N" else b[:, :n]
    c = make(n, m)
    c0 = c.clone()
    torch.cuda.synchronize()
    for _ in range(2):   # the second call's preparation overlaps the first call's product
        c.copy_(c0)
        torch.cuda.synchronize()
        dev.dgemm_ozaki(ta, tb, m, n, k, -1.0, a, a.shape[1], b, b.shape[1], 1.0, c, m, want_slices=False)
        dev.dgemm_ozaki(ta, tb, m, n, k, 1.0, a, a.shape[1], b, b.shape[1], 1.0, c, m, want_slices=False)
        dev.dgemm_ozaki(ta, tb, m, n, k, 1.0, a, a.shape[1], b, b.shape[1], 0.0, c, m, want_slices=False)
        dev.sync()
    ref = opa @ opb
    assert float((c.T - ref).norm()) <= 2e-14 * float(ref.norm())
