"""GPU parity of the DGER, DSYMV and DTRSV kernels at the sizes where their
dispatch changes, on device operands against plain 64-bit torch.

* DGER: 512-row x 32-column tiles, 128-bit rows only for 16-byte aligned
  columns, columns of a zero y_j skipped.  One FMA per element: the error of
  an element is at most one rounding of each of alpha y_j, the product and
  the sum on either side, 4 x 2^-53 x 2.5 (|A| <= 1, |alpha x y| <= 0.5 on
  the test's inputs) < 2e-15.
* DSYMV: 64 x 64 tiles, four threads per row in the final sum; n rounded
  sums of n products: n 2^-53 |A||x| <= n^2 2^-53 / 4 per element as a
  bound, 1e-13 relative to the result's norm as in the other DSYMV tests.
* DTRSV: 64-row blocks; the 25th and later fold the block before into the
  inverse; more blocks than SMs means several blocks per CTA.  Residual
  ||op(A) x - b|| / (||A|| ||x||) <= 1e-14, as in the other DTRSV tests.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import libgpublas_gb300 as g
    d = g.Device(0)
    yield d
    d.close()


def uni(gen, *shape):
    import torch
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1


def gen_of(seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("m", [1, 2, 255, 257, 511, 512, 513, 1025])
@pytest.mark.parametrize("n", [1, 7, 32, 33, 71])
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (2, 0), (2, 1)])
def test_dger_tiles(dev, m, n, pad, shift):
    import torch
    gen = gen_of(m * 1000 + n)
    ld = m + pad
    buf = uni(gen, n * ld + shift)
    x, y = uni(gen, m), uni(gen, n)
    if n > 5:
        y[3] = 0.0
        y[5] = -0.0
        x[0] = float("inf")    # not propagated into the columns of a zero y_j
    a0 = buf[shift:].view(n, ld).clone()
    torch.cuda.synchronize()
    st = dev.L.gbx_dger(dev.ctx, m, n, -0.5, p(x), 1, p(y), 1, C.c_void_p(buf.data_ptr() + 8 * shift), ld)
    assert st == 0
    dev.sync()
    got = buf[shift:].view(n, ld)
    ref = a0.clone()
    live = y != 0
    ref[live, :m] += (-0.5 * y[live])[:, None] * x[None, :]
    assert torch.equal(got[:, m:], a0[:, m:])
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(got), fin)
    assert float((got[fin] - ref[fin]).abs().max()) <= 2e-15


@pytest.mark.parametrize("n", [127, 128, 129, 513])
@pytest.mark.parametrize("uplo", "UL")
def test_dsymv_tiles(dev, n, uplo):
    import torch
    gen = gen_of(n)
    a, x, y = uni(gen, n, n), uni(gen, n), uni(gen, n)
    am = a.T
    sym = am.tril() + am.tril(-1).T if uplo == "L" else am.triu() + am.triu(1).T
    ref = 1.5 * (sym @ x) - 0.5 * y
    torch.cuda.synchronize()
    assert dev.L.gbx_dsymv(dev.ctx, uplo.encode(), n, 1.5, p(a), n, p(x), 1, -0.5, p(y), 1) == 0
    dev.sync()
    assert float((y - ref).norm()) <= 1e-13 * float(ref.norm())


@pytest.mark.parametrize("n", [65, 1535, 1536, 1537, 1601, 9729, 9800])
@pytest.mark.parametrize("uplo", "UL")
@pytest.mark.parametrize("trans", "NT")
def test_dtrsv_blocks(dev, n, uplo, trans):
    import torch
    gen = gen_of(n)
    ld = n + 1
    a = uni(gen, n, ld) / n
    a.diagonal().copy_(torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) + 1)
    b = uni(gen, n)
    inc = 2
    x = torch.full((n * inc,), 7.0, dtype=torch.float64, device="cuda")
    x[::inc] = b
    torch.cuda.synchronize()
    diag = "U" if n % 2 else "N"
    st = dev.L.gbx_dtrsv(dev.ctx, uplo.encode(), trans.encode(), diag.encode(), n, p(a), ld, p(x), inc)
    assert st == 0
    dev.sync()
    t = a[:, :n].T
    t = t.tril() if uplo == "L" else t.triu()
    if diag == "U":
        t = t.clone()
        t.diagonal().fill_(1.0)
    op = t if trans == "N" else t.T
    got = x[::inc]
    assert float((op @ got - b).norm()) <= 1e-14 * float(op.norm()) * float(got.norm())
    assert bool((x[1::inc] == 7.0).all())
