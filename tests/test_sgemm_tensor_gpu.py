"""GPU parity of SGEMM on the tensor cores (bf16 split) against 64-bit torch,
at the edges of its tiles (128 x 128, 64 values of k per block, one or two
blocks per accumulator) and for the operands it leaves to the SIMT kernel.

Tolerance, per element, in units of 2^-24 sum_k |a_ik b_kj| (|alpha| = 1):
the products left out 1; truncated accumulation of the large products, at most
8 steps of one unit (2 ulp of the partial sum) each in an accumulator, 16; the
small products' accumulators are 2^-8 of that per step, k/16 x 5 steps x 2 x
2^-8 < k / 400; the FP32 sums of the accumulators k / 64 + 3; and the final
alpha acc + beta C two roundings of the result.  In all 24 + k / 48, plus
2 units of |beta C| + |result|.  The SIMT kernel: k + 4 units."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


@pytest.fixture(scope="module")
def dev():
    import libgpublas_gb300 as g
    d = g.Device(0)
    yield d
    d.close()


def rand(gen, *s):
    import torch
    return torch.rand(*s, device="cuda", generator=gen) * 2 - 1


def gen_of(seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def call(dev, ta, tb, m, n, k, alpha, a, b, beta, c):
    import torch
    torch.cuda.synchronize()
    st = dev.L.gbx_sgemm(dev.ctx, ta.encode(), tb.encode(), m, n, k, alpha, C.c_void_p(a.data_ptr()), a.shape[1],
                         C.c_void_p(b.data_ptr()), b.shape[1], beta, C.c_void_p(c.data_ptr()), c.shape[1])
    assert st == 0
    dev.sync()


def operands(gen, ta, tb, m, n, k, pad):
    a = rand(gen, *((k, m + pad) if ta == "N" else (m, k + pad)))
    b = rand(gen, *((n, k + pad) if tb == "N" else (k, n + pad)))
    opa = a[:, :m].T if ta == "N" else a[:, :k]
    opb = b[:, :k].T if tb == "N" else b[:, :n]
    return a, b, opa, opb


def check(got, c0, opa, opb, alpha, beta, units):
    ref = alpha * (opa.double() @ opb.double()) + (beta * c0.double() if beta else 0.0)
    mag = opa.double().abs() @ opb.double().abs()
    tol = U * (units * mag + 2 * ref.abs() + (2 * abs(beta) * c0.double().abs() if beta else 0.0)) + 1e-44
    bad = (got.double() - ref).abs() > tol
    assert not bool(bad.any()), float(((got.double() - ref).abs() / tol).max())


SHAPES = [(1024, 1024, 16), (1000, 1100, 8), (640, 640, 63), (700, 900, 64), (700, 900, 65), (127, 129, 1024),
          (128, 128, 1025), (129, 255, 1100), (1, 4096, 1024), (4096, 1, 1024), (257, 640, 255), (257, 640, 256),
          (257, 640, 257), (513, 385, 321), (2049, 2000, 130)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("ta,tb", ["NN", "TN", "NT", "TT"])
def test_edges(dev, m, n, k, ta, tb):
    import torch
    dev.L.gbx_sgemm_tensor_choice.argtypes = [C.c_int] * 4
    assert dev.L.gbx_sgemm_tensor_choice(m, n, k, 152) == 1
    pad = m % 3
    gen = gen_of(m + n + k)
    a, b, opa, opb = operands(gen, ta, tb, m, n, k, pad)
    for alpha, beta in [(1.0, 0.0), (-1.0, 0.5)]:
        c = rand(gen, n, m + pad)
        if beta == 0.0:
            c[:, :m] = float("nan")   # overwritten, not scaled
        c0 = c.clone()
        call(dev, ta, tb, m, n, k, alpha, a, b, beta, c)
        assert torch.equal(c[:, m:], c0[:, m:])
        check(c[:, :m].T, c0[:, :m].T, opa, opb, alpha, beta, 24 + k / 48)


@pytest.mark.parametrize("which", "ab")
@pytest.mark.parametrize("value", ["inf", "-inf", "nan", "1e-20", "1e25", "1e-41"])
def test_uncovered_values(dev, which, value):
    """One element outside the split's range: the result is the SIMT core's."""
    import torch
    m, n, k = 400, 500, 300
    gen = gen_of(7)
    a, b, opa, opb = operands(gen, "N", "N", m, n, k, 0)
    (a if which == "a" else b)[17, 23] = float(value)
    c = rand(gen, n, m)
    c0 = c.clone()
    call(dev, "N", "N", m, n, k, 1.0, a, b, 0.5, c)
    ref = opa.double() @ opb.double() + 0.5 * c0.T.double()
    got = c.T
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    assert torch.equal(got[torch.isinf(ref)].sign(), ref[torch.isinf(ref)].sign().float())
    fin = torch.isfinite(ref)
    tol = U * ((k + 4) * (opa.double().abs() @ opb.double().abs()) + 2 * ref.abs() + c0.T.double().abs())
    assert bool(((got.double() - ref).abs() <= tol)[fin].all())
    # the next call on the same context, with covered operands, is the tensor kernel's again
    (a if which == "a" else b)[17, 23] = 0.5
    c = c0.clone()
    call(dev, "N", "N", m, n, k, 1.0, a, b, 0.5, c)
    check(c.T, c0.T, a.T, b.T, 1.0, 0.5, 24 + k / 48)


def test_wide_exponents(dev):
    """Magnitudes over 2^-60 .. 2^60 keep the elementwise bound."""
    import torch
    m, n, k = 512, 400, 640
    gen = gen_of(3)
    a, b, opa, opb = operands(gen, "T", "N", m, n, k, 0)
    for x, s in ((a, 0), (b, 1)):
        e = torch.randint(-30, 31, x.shape, device="cuda", generator=gen)
        x.copy_(torch.ldexp(x.sign() * (x.abs() * 0.5 + 0.5), e))
    c = torch.zeros(n, m, device="cuda")
    call(dev, "T", "N", m, n, k, 1.0, a, b, 0.0, c)
    check(c.T, c.T, opa, opb, 1.0, 0.0, 24 + k / 48)


def test_operands_larger_than_the_workspace_limit(dev):
    """The planes of this product would take more than 2 GiB: computed in pieces."""
    m, n, k = 1300, 300, 230000
    gen = gen_of(5)
    a, b, opa, opb = operands(gen, "T", "N", m, n, k, 0)
    c = rand(gen, n, m)
    c0 = c.clone()
    call(dev, "T", "N", m, n, k, 1.0, a, b, 0.5, c)
    check(c.T, c0.T, opa, opb, 1.0, 0.5, 24 + k / 48)


def test_first_call_under_capture_takes_the_simt_core():
    """A capture must not allocate: without the planes' workspace the call is
    recorded as the SIMT kernel, and its replay computes the product."""
    import torch
    import libgpublas_gb300 as g
    d = g.Device(0)
    m, n, k = 512, 512, 512
    gen = gen_of(11)
    a, b, opa, opb = operands(gen, "N", "N", m, n, k, 0)
    c = torch.zeros(n, m, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    d.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        assert d.L.gbx_sgemm(d.ctx, b"N", b"N", m, n, k, 1.0, C.c_void_p(a.data_ptr()), m, C.c_void_p(b.data_ptr()),
                             k, 0.0, C.c_void_p(c.data_ptr()), m) == 0
    graph.replay()
    torch.cuda.synchronize()
    check(c.T, c.T, opa, opb, 1.0, 0.0, k + 4)
    d.set_stream(None)
    d.close()
