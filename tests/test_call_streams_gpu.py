"""A stream of equal calls takes no longer per call than one call on its own.

A call that overlaps the one before may be placed on the SMs while that one
runs; it must not end up unevenly on them.  Compared: the shortest of several
runs of one call between two events, and of 100 calls, per call.  A kernel of
the same work placed evenly takes the same time in both; the events add to the
single call, so the stream is allowed a fifth more than that."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
CALLS = 100


def _per_call(dev, call, count, runs):
    import torch
    stream = torch.cuda.ExternalStream(dev.stream())
    best = float("inf")
    for _ in range(runs):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record(stream)
        call(count)
        b.record(stream)
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / count)
    return best


def _check(dev, call):
    call(CALLS)
    alone, many = _per_call(dev, call, 1, 20), _per_call(dev, call, CALLS, 5)
    assert many <= 1.2 * alone, f"{1e3 * many:.1f} us a call in a stream, {1e3 * alone:.1f} us alone"


@pytest.mark.parametrize("m,n,k", [(64, 64, 512), (64, 128, 512), (96, 128, 256), (96, 128, 512), (128, 128, 512),
                                   (128, 128, 2048), (128, 152, 512), (128, 304, 512)])
@pytest.mark.parametrize("ta", ["N", "T"])
def test_dgemm(dev, m, n, k, ta):
    import torch
    import libgpublas_gb300 as g
    a, b = (torch.rand(k * max(m, n), dtype=torch.float64, device="cuda") for _ in range(2))
    c = torch.rand(m * n, dtype=torch.float64, device="cuda")
    ops = (g.GbxOp * CALLS)(*[g.GbxOp(kind=1, transa=ta.encode(), transb=b"N", m=m, n=n, k=k, alpha=1.0, beta=0.5,
                                      A=a.data_ptr(), lda=m if ta == "N" else k, B=b.data_ptr(), ldb=k,
                                      C=c.data_ptr(), ldc=m) for _ in range(CALLS)])
    _check(dev, lambda count: dev.ops_run(ops, count))


def test_sgemm(dev):
    import torch
    m, n, k = 128, 128, 900
    a, b, c = (torch.rand(k * n, device="cuda") for _ in range(3))
    args = (dev.ctx, b"N", b"N", m, n, k, C.c_float(1.0), C.c_void_p(a.data_ptr()), m, C.c_void_p(b.data_ptr()), k,
            C.c_float(0.5), C.c_void_p(c.data_ptr()), m)

    def call(count):
        for _ in range(count):
            assert dev.L.gbx_sgemm(*args) == 0
    _check(dev, call)


@pytest.mark.parametrize("m,n", [(300, 4000), (1000, 800)])
def test_dger(dev, m, n):
    import torch
    a = torch.rand(m * n, dtype=torch.float64, device="cuda")
    x, y = torch.rand(m, dtype=torch.float64, device="cuda"), torch.rand(n, dtype=torch.float64, device="cuda")
    args = (dev.ctx, m, n, C.c_double(1e-9), C.c_void_p(x.data_ptr()), 1, C.c_void_p(y.data_ptr()), 1,
            C.c_void_p(a.data_ptr()), m)

    def call(count):
        for _ in range(count):
            assert dev.L.gbx_dger(*args) == 0
    _check(dev, call)
