"""Which kernel an SGEMM's result comes from, by its rounding: for random operands
and k = 4096 the tensor cores leave a relative Frobenius error near 1.5e-7 (FP32
sums of accumulators of 128 terms), the SIMT core's single chains of 4096
roundings near 1.1e-6 (sqrt(k) 2^-24 / 3 and up).  4e-7 lies between; it does not
depend on the operands' scales, up to the ends of the range that the split covers:
magnitudes in 2^-90 .. 2^60, and none below 2^-34 beside an operand that goes below
2^-60.  Products of lower terms are subnormal there, or sums near the top of the
format."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
M, N, K = 256, 384, 4096
LIMIT = 4e-7


def error(dev, a, b):
    import torch
    c = torch.empty(N, M, device="cuda")
    torch.cuda.synchronize()
    assert dev.L.gbx_sgemm(dev.ctx, b"N", b"N", M, N, K, C.c_float(1.0), C.c_void_p(a.data_ptr()), M,
                           C.c_void_p(b.data_ptr()), K, C.c_float(0.0), C.c_void_p(c.data_ptr()), M) == 0
    dev.sync()
    ref = b.double() @ a.double()
    return float((c.double() - ref).norm() / ref.norm())


def operand(seed, rows, cols, lo):
    """Magnitudes in [2^lo, 2^(lo + 1)), random signs."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    v = 1 + torch.rand(rows, cols, device="cuda", generator=gen)
    v.clamp_(max=2 - 2.0 ** -20)
    return torch.ldexp(v * (torch.rand(rows, cols, device="cuda", generator=gen) < 0.5).float().mul(2).sub(1),
                       torch.tensor(lo, device="cuda"))


@pytest.mark.parametrize("ea,eb", [(0, 0), (-60, 0), (-60, 59), (-50, -50), (-31, -31), (30, 30), (59, 59),
                                   (59, -59), (-90, 59), (59, -90), (-90, 0), (-90, -34), (-34, -90), (-60, -60),
                                   (-60, -35)])
def test_covered_range_on_the_tensor_cores(dev, ea, eb):
    assert error(dev, operand(1, K, M, ea), operand(2, N, K, eb)) < LIMIT


@pytest.mark.parametrize("ea,eb", [(-61, -35), (-35, -61), (-90, -35), (-61, -61), (-91, 0), (0, -91), (-91, 59)])
def test_other_ranges_on_the_simt_core(dev, ea, eb):
    assert LIMIT < error(dev, operand(1, K, M, ea), operand(2, N, K, eb)) < 4e-6


@pytest.mark.parametrize("which", "ab")
@pytest.mark.parametrize("value", [2.0 ** -90 * (1 - 2.0 ** -24), -2.0 ** -91, 2.0 ** 60 * (1 + 2.0 ** -23)])
def test_outside_it_on_the_simt_core(dev, which, value):
    a, b = operand(3, K, M, 0), operand(4, N, K, 0)
    assert error(dev, a, b) < LIMIT
    x = a if which == "a" else b
    keep = float(x[5, 7])
    x[5, 7] = value if abs(value) < 1 else 2.0 ** 60 * (1 + 2.0 ** -23) * (1 if value > 0 else -1)
    err = error(dev, a, b)
    if abs(value) < 1:   # (a large one is the result's only part that counts)
        assert LIMIT < err < 4e-6
    x[5, 7] = keep
    assert error(dev, a, b) < LIMIT   # and back


@pytest.mark.parametrize("value", [2.0 ** -90, 2.0 ** 60, 0.0, -0.0])
def test_the_range_includes_its_ends(dev, value):
    a, b = operand(5, K, M, 0), operand(6, N, K, 0)
    if value > 1:   # all of them: otherwise one column's error is the whole one
        a = a.sign() * value
    else:
        a[5, 7] = value
    assert error(dev, a, b) < LIMIT


def test_captured_calls_on_the_simt_core(dev):
    import torch
    import libgpublas_gb300 as g
    d = g.Device(0)
    a, b, c = operand(7, K, M, 0), operand(8, N, K, 0), torch.empty(N, M, device="cuda")
    assert error(d, a, b) < LIMIT
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    d.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        assert d.L.gbx_sgemm(d.ctx, b"N", b"N", M, N, K, C.c_float(1.0), C.c_void_p(a.data_ptr()), M,
                             C.c_void_p(b.data_ptr()), K, C.c_float(0.0), C.c_void_p(c.data_ptr()), M) == 0
    d.set_stream(None)
    graph.replay()
    torch.cuda.synchronize()
    ref = b.double() @ a.double()
    assert LIMIT < float((c.double() - ref).norm() / ref.norm()) < 4e-6
    d.close()
