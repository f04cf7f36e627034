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
