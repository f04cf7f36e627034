"""Streams of DGEMMs and DTRSMs each of which reads the one before, at sizes whose
launches overlap it: at most one CTA per SM of the core's 16, 32 and 64 tiles.

Tolerance: an orthogonal factor, so a product of length n adds at most (n + 4) u
relative to the norm; DTRSM with a diagonal of 2 and a norm below 3 adds 20 n u."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
CALLS = 30


def few_tiles(lib, bm, sms):
    """The largest square C that is cut into tiles of bm, one CTA per SM at most."""
    f = lib.gbx_dgemm_tile_choice
    f.argtypes = [C.c_int] * 4
    for n in range(2000, 32, -1):
        if f(n, n, 0, sms) == bm and (-(-n // bm)) ** 2 <= sms:
            return n
    return 0


@pytest.mark.parametrize("bm", [16, 32, 64])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_products(dev, bm, trans):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = few_tiles(dev.L, bm, sms)
    if not n:
        pytest.skip("no such launch")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    q = torch.linalg.qr(torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) - 0.5)[0].contiguous()
    c = [torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) for _ in range(2)]
    ref = c[0].clone()
    torch.cuda.synchronize()
    for i in range(CALLS):   # the buffers take turns: a call also overwrites what the one before has read
        assert dev.dgemm("N", trans, n, n, n, 1.0, c[i % 2], n, q, n, 0.0, c[(i + 1) % 2], n) == 0
    dev.sync()
    # column-major: C^T = op(Q)^T C^T on the tensors
    for _ in range(CALLS):
        ref = (q if trans == "N" else q.T) @ ref
    got = c[CALLS % 2]
    assert float((got - ref).norm()) <= CALLS * (n + 4) * 2.0 ** -53 * float(ref.norm())


@pytest.mark.parametrize("n,rhs", [(130, 16), (200, 64), (500, 96), (1000, 16)])
def test_solves(dev, n, rhs):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    a = (torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1) / n
    a.diagonal().copy_(torch.full((n,), 2.0, dtype=torch.float64, device="cuda"))
    x = torch.rand(rhs, n, dtype=torch.float64, device="cuda", generator=gen)   # column-major n x rhs
    ref = x.T.clone()
    torch.cuda.synchronize()
    for i in range(6):
        dev.dtrsm("L", "LU"[i % 2], "N", "N", n, rhs, 2.0, a, n, x, n)
    dev.sync()
    am = a.T
    for i in range(6):
        ref = torch.linalg.solve_triangular(am, 2.0 * ref, upper=i % 2 == 1)
    assert float((x.T - ref).norm()) <= 6 * 20 * n * 2.0 ** -53 * float(ref.norm())
