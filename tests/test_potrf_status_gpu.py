"""gbx_dpotrf_small after a call that left an error in the context's status word:
the factorisation waits for its own warps all the same and is right (bit for bit
what it is otherwise), and the error is that of the earlier call."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 100, 256])
def test_factor_after_a_reported_error(n):
    import torch
    import libgpublas_gb300 as g
    dev = g.Device(0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a, b, c = uni(256, 256), uni(256, 256), uni(256, 256)
    a[3, 5] = float("inf")
    w = uni(n, n)
    spd = w @ w.T + n * torch.eye(n, dtype=torch.float64, device="cuda")
    want, got = spd.clone(), [spd.clone() for _ in range(4)]
    info = torch.full((5,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dev.dpotrf_small(n, want, n, info)
    dev.sync()
    dev.dgemm_ozaki("N", "N", 256, 256, 256, 1.0, a, 256, b, 256, 0.0, c, 256, want_slices=False)
    for i, x in enumerate(got):
        dev.dpotrf_small(n, x, n, info[i + 1:])
    assert dev.L.gbx_ctx_sync(dev.ctx) != 0 and "non-finite" in dev.last_error()
    assert info.tolist() == [0] * 5
    for x in got:
        assert torch.equal(x, want)
    dev.close()
