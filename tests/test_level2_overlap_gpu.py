"""Level 2 calls that overlap the call before: short streams of dependent DGEMV,
DGER and DSYMV calls, sizes around the partials' rows (64) and chunks (16 columns)
and around one CTA per SM, the limit of the overlap (152 SMs).

Tolerance: a product of k terms is within (k + 4) u of |A| |x| in the 2-norm, an
update within 2 u; the vectors are scaled to norm 1 and the updates by 1/4, so
that an error grows by less than 2 in the four rounds and |A| by less than 4:
64 (max(m, n) + 8) u relative to the norm of the first A."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (63, 15), (64, 16), (65, 17), (130, 33), (300, 1215), (300, 1216), (300, 4000),
                                 (512, 4864), (513, 4865), (1000, 800), (9000, 40), (9729, 31)])
def test_reflectors(dev, m, n):
    import torch
    from libgpublas_gb300._lib import _dp
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a = uni(n, m)   # column-major m x n
    a /= a.norm()
    norm0 = 1.0
    us, vs = uni(4, n), uni(4, m)
    us /= us.norm(dim=1, keepdim=True)
    vs /= vs.norm(dim=1, keepdim=True)
    ref = a.T.clone()
    ws = torch.zeros(4, m, dtype=torch.float64, device="cuda")
    ts = torch.zeros(4, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for i in range(4):
        u, v, w, t = us[i], vs[i], ws[i], ts[i]
        dev.dgemv("T", m, n, 1.0, a, m, v, 1, 0.0, t, 1)
        assert dev.L.gbx_dger(dev.ctx, m, n, -0.25, _dp(v), 1, _dp(t), 1, _dp(a), m) == 0
        dev.dgemv("N", m, n, 1.0, a, m, u, 1, 0.0, w, 1)
        assert dev.L.gbx_dger(dev.ctx, m, n, -0.25, _dp(w), 1, _dp(u), 1, _dp(a), m) == 0
    dev.sync()
    tol = 64 * (max(m, n) + 8) * 2.0 ** -53 * norm0
    for i in range(4):
        rt = ref.T @ vs[i]
        assert float((ts[i] - rt).norm()) <= tol
        ref -= 0.25 * torch.outer(vs[i], rt)
        rw = ref @ us[i]
        assert float((ws[i] - rw).norm()) <= tol
        ref -= 0.25 * torch.outer(rw, us[i])
    assert float((a.T - ref).norm()) <= tol


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 1088, 1089, 1153])
@pytest.mark.parametrize("uplo", "UL")
def test_symmetric_products(dev, n, uplo):
    """x, A x, A (A x), ..: each call reads the one before."""
    import torch
    from libgpublas_gb300._lib import _dp
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    a = torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a = a + a.T
    a /= a.norm()
    x = torch.rand(5, n, dtype=torch.float64, device="cuda", generator=gen)
    x[0] /= x[0].norm()
    torch.cuda.synchronize()
    for i in range(4):
        assert dev.L.gbx_dsymv(dev.ctx, uplo.encode(), n, 1.0, _dp(a), n, _dp(x[i]), 1, 0.0, _dp(x[i + 1]), 1) == 0
    dev.sync()
    ref = x[0].clone()
    for i in range(4):
        ref = a @ ref
        assert float((x[i + 1] - ref).norm()) <= 64 * (n + 8) * 2.0 ** -53


@pytest.mark.parametrize("m,n", [(1, 9), (255, 8), (256, 9), (257, 33), (300, 1208), (511, 1209), (512, 2424), (513, 608),
                                 (1000, 609), (1000, 1217), (700, 4865)])
@pytest.mark.parametrize("pad", [0, 1])
def test_update_widths(dev, m, n, pad):
    """8, 16 or 32 columns per CTA, second rows that end inside a CTA, columns
    left alone (y_j = 0).  Two roundings of values below 2: 2^-51."""
    import torch
    from libgpublas_gb300._lib import _dp
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7 * m + n + pad)

    def uni(*s):
        return torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a, x, y = uni(n, m + pad), uni(m), uni(n)
    y[torch.rand(n, device="cuda", generator=gen) < 0.2] = 0.0
    a[y == 0.0, 0] = float("inf")
    ref = a.clone()
    live = y != 0.0
    ref[live, :m] += 0.75 * y[live][:, None] * x[None, :]
    torch.cuda.synchronize()
    assert dev.L.gbx_dger(dev.ctx, m, n, 0.75, _dp(x), 1, _dp(y), 1, _dp(a), m + pad) == 0
    dev.sync()
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(a), fin)
    assert torch.equal(a[~live], ref[~live]) and torch.equal(a[:, m:], ref[:, m:])
    assert float((a[fin] - ref[fin]).abs().max()) <= 2.0 ** -51
