"""Calls recorded in a CUDA graph, those that overlap the call before and the
cooperative DTRSV among them: a replay gives the bits of the same calls made
directly."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def own():
    import libgpublas_gb300 as g
    d = g.Device(0)
    yield d
    d.set_stream(None)
    d.close()


def p(t):
    return C.c_void_p(t.data_ptr())


def capture(dev, calls):
    import torch
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    dev.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        calls()
    dev.set_stream(None)
    return graph


def uni(seed, *s):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1


@pytest.mark.parametrize("n", [70, 1000])
def test_dtrsv_after_dtrsm(own, n):
    """The context has never run a DTRSV: the workspace of a DTRSM of the order is enough."""
    import torch
    import libgpublas_gb300 as g
    a = uni(1, n, n) / n + 2 * torch.eye(n, dtype=torch.float64, device="cuda")
    b, x, y = uni(2, 64, n), uni(3, n), uni(3, n)
    torch.cuda.synchronize()
    own.dtrsm("L", "L", "N", "N", n, 64, 1.0, a, n, b, n)
    own.sync()

    def solve(d, v):
        assert d.L.gbx_dtrsv(d.ctx, b"L", b"N", b"N", n, p(a), n, p(v), 1) == 0
    graph = capture(own, lambda: solve(own, x))
    graph.replay()
    torch.cuda.synchronize()
    other = g.Device(0)
    solve(other, y)
    other.sync()
    other.close()
    assert torch.equal(x, y)


def test_reduction_after_a_shorter_one(own):
    """A context that has run a reduction of one block can capture one of any size."""
    import torch
    x = uni(10, 1 << 20)
    r = torch.zeros(2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    own.dnrm2(100, x, 1, r)
    own.sync()
    graph = capture(own, lambda: own.ddot(1 << 20, x, 1, x, 1, r[1:]))
    graph.replay()
    torch.cuda.synchronize()
    want = torch.zeros(1, dtype=torch.float64, device="cuda")
    own.ddot(1 << 20, x, 1, x, 1, want)
    own.sync()
    assert torch.equal(r[1:], want)


def test_a_sequence_of_calls(own):
    import torch
    n, m = 300, 200
    a0, l, k = uni(4, n, n), uni(5, n, n) / n + 2 * torch.eye(n, dtype=torch.float64, device="cuda"), uni(6, n, m)
    spd0 = 4 * torch.eye(256, dtype=torch.float64, device="cuda") + uni(7, 256, 256) / 64
    spd0 = (spd0 + spd0.T).contiguous()
    v0, w0 = uni(8, n), uni(9, n)
    state = [t.clone() for t in (a0, k, spd0, v0, w0)]
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    idx = torch.zeros(2, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")

    def reset():
        for t, z in zip(state, (a0, k, spd0, v0, w0)):
            t.copy_(z)
        out.zero_(), idx.zero_()
        torch.cuda.synchronize()

    def calls():
        a, b, spd, v, w = state
        L, ctx = own.L, own.ctx
        one, zero, small = C.c_double(1.0), C.c_double(0.0), C.c_double(1e-3)
        for st in (L.gbx_dgemv(ctx, b"N", n, n, small, p(a), n, p(v), 1, one, p(w), 1),
                   L.gbx_dger(ctx, n, n, small, p(v), 1, p(w), 1, p(a), n),
                   L.gbx_dgemv(ctx, b"T", n, n, small, p(a), n, p(w), 1, one, p(v), 1),
                   L.gbx_dsymv(ctx, b"L", n, small, p(a), n, p(v), 1, one, p(w), 1),
                   L.gbx_dtrsv(ctx, b"L", b"T", b"N", n, p(l), n, p(w), 1),
                   L.gbx_daxpy(ctx, n, small, p(w), 1, p(v), 1),
                   L.gbx_dscal(ctx, n, C.c_double(0.5), p(v), 1),
                   L.gbx_ddot(ctx, n, p(v), 1, p(w), 1, p(out)),
                   L.gbx_dnrm2(ctx, n, p(v), 1, p(out[1:])),
                   L.gbx_ddot(ctx, n * m, p(b), 1, p(b), 1, p(out[2:])),
                   L.gbx_dnrm2(ctx, n * m, p(b), 1, p(out[3:])),
                   L.gbx_idamax(ctx, n * n, p(a), 1, p(idx)),
                   L.gbx_idamin(ctx, n, p(w), 1, p(idx[1:])),
                   L.gbx_dgemm(ctx, b"N", b"T", n, n, m, small, p(b.view(-1)), n, p(b.view(-1)), n, one, p(a), n),
                   L.gbx_dtrsm(ctx, b"R", b"L", b"T", b"N", m, n, one, p(l), n, p(b), m)):
            assert st == 0
        own.dpotrf_small(256, spd, 256, info)
        own.dgemm_ozaki("N", "N", 256, 256, 256, 1e-3, spd, 256, spd, 256, 1.0, a, n, want_slices=False)

    reset()
    calls()
    own.sync()
    want = [t.clone() for t in (*state, out, idx)]
    graph = capture(own, calls)
    for _ in range(3):
        reset()
        graph.replay()
        torch.cuda.synchronize()
        for got, ref in zip((*state, out, idx), want):
            assert torch.equal(got, ref)
    assert int(info) == 0
