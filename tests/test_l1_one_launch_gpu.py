"""GPU parity of the one-launch reductions (DDOT, DNRM2, IDAMAX, IDAMIN) at
the sizes where their grid changes: one block (n <= 512), two, and the full
grid of 608 blocks, aligned and not, back to back on one context (each launch
leaves the count of finished blocks at zero for the next, and overlaps the end
of the one before).  DDOT: n rounded products and sums, n 2^-53 sum |x y|; DNRM2:
4 x 2^-53 sqrt(n) relative is above its n / (2 x 155648) sequential roundings
per thread and the tree; indices exactly."""
import math

import pytest

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 511, 512, 513, 1025, 10001, 311295, 311296, 311297, 622593, 3000001]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift", [0, 1])
def test_reductions(n, shift):
    import torch
    import libgpublas_gb300 as g
    dev = g.Device(0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = (torch.rand(n + 1, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1)[shift:n + shift]
    y = (torch.rand(n + 1, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1)[shift:n + shift]
    a, b = n // 3, (2 * n) // 3
    if n > 10:   # tied maxima and minima, in different blocks where there are several
        x[a], x[b] = -2.0, 2.0
        x[a + 1], x[b + 1] = 0.0, -0.0
    dot, nrm = (torch.zeros(3, dtype=torch.float64, device="cuda") for _ in range(2))
    imax, imin = (torch.zeros(3, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for r in range(3):
        dev.ddot(n, x, 1, y, 1, dot[r:])
        dev.dnrm2(n, x, 1, nrm[r:])
        dev.idamax(n, x, 1, imax[r:])
        dev.idamin(n, x, 1, imin[r:])
    dev.sync()
    for t in (dot, nrm, imax, imin):
        assert torch.equal(t, t[:1].expand(3))
    assert abs(float(dot[0] - (x * y).sum())) <= n * 2.0 ** -52 * float((x * y).abs().sum())
    assert abs(float(nrm[0] - x.norm())) <= 4 * 2.0 ** -53 * math.sqrt(n) * float(x.norm())
    assert int(imax[0]) == int(x.abs().argmax()) + 1 or n > 10
    if n > 10:
        assert int(imax[0]) == a + 1 and int(imin[0]) == a + 2
    dev.close()


@pytest.mark.parametrize("n", [512, 1025, 311297])
@pytest.mark.parametrize("value", [1e-300, 1e300, 1e-320])
def test_dnrm2_one_element_out_of_range(n, value):
    """A single very small or large element, in the last block."""
    import torch
    import libgpublas_gb300 as g
    dev = g.Device(0)
    for rest in (0.0, abs(value)):
        x = torch.full((n,), rest, dtype=torch.float64, device="cuda")
        x[n - 1] = value
        r = torch.zeros(1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        dev.dnrm2(n, x, 1, r)
        dev.sync()
        want = abs(value) * (math.sqrt(n) if rest else 1.0)
        assert abs(float(r) - want) <= 1e-13 * want + 5e-324
    dev.close()
