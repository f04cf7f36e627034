"""gbx_dpotrf_small and the triangular inverse inside gbx_dtrsm_ozaki at the
edges of their 32-row blocks, and over the exponent range of the pivots'
reciprocal (an approximate reciprocal refined once, and a division near the
ends of the range).

Tolerances: the Cholesky factor of a matrix with condition number below 10
is within 10 n 2^-53 of the exact one per entry, relative to the diagonal (a
few rounded operations per entry and step); a 2 x 2 factor within 8 x 2^-53.
The inverse is seen through B = I in DTRSM: every entry within 16 n 2^-53 of
the 64-bit inverse of a well-conditioned triangle plus the product's 1e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 33, 39, 40, 41, 72, 95, 96, 97, 224, 255])
def test_potrf_blocks(dev, n):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    w = torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a0 = w @ w.T + n * torch.eye(n, dtype=torch.float64, device="cuda")
    lda = n + 3
    A = torch.zeros(n, lda, dtype=torch.float64, device="cuda")
    A[:, :n] = a0
    info = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):   # the second factorisation follows the first on the stream
        A[:, :n] = a0
        torch.cuda.synchronize()
        dev.dpotrf_small(n, A, lda, info)
        dev.sync()
    assert int(info) == 0
    got = A[:, :n].T.tril()
    ref = torch.linalg.cholesky(a0)
    assert float((got - ref).abs().max()) <= 10 * n * 2.0 ** -53 * float(ref.diagonal().max())


@pytest.mark.parametrize("e", [-1070, -1021, -1000, -996, -500, 0, 500, 976, 1000, 1016])
def test_potrf_pivot_range(dev, e):
    import torch
    s = 2.0 ** e
    a = np.array([[1.0, 0.3], [0.3, 0.8]])
    A = torch.from_numpy(a * s).cuda()
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dev.dpotrf_small(2, A, 2, info)
    dev.sync()
    assert int(info) == 0
    # the reference on the scaled values (subnormal inputs are rounded), in extended range
    b = (a * s).astype(np.longdouble)
    l00 = np.sqrt(b[0, 0])
    l10 = b[1, 0] / l00
    l11 = np.sqrt(b[1, 1] - l10 * l10)
    got = A.cpu().numpy().T
    tol = 8 * 2.0 ** -53 + (2.0 ** -1074 / s) * 4   # and the subnormal spacing of the intermediate products
    for g, r in ((got[0, 0], l00), (got[1, 0], l10), (got[1, 1], l11)):
        assert abs(g - float(r)) <= tol * abs(float(r))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 129, 255, 256])
@pytest.mark.parametrize("uplo", "UL")
@pytest.mark.parametrize("trans", "NT")
def test_inverse_blocks(dev, n, uplo, trans):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    t = (torch.rand(n, n + 2, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1) / n
    t.diagonal().copy_(torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) + 1)
    diag = "U" if n % 2 else "N"
    B = torch.eye(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    dev.dtrsm_ozaki("L", uplo, trans, diag, n, n, 1.0, t, n + 2, B, n)
    dev.sync()
    m = t[:, :n].T
    m = m.tril() if uplo == "L" else m.triu()
    if diag == "U":
        m = m.clone()
        m.diagonal().fill_(1.0)
    op = m if trans == "N" else m.T
    ref = torch.linalg.inv(op)
    assert float((B.T - ref).abs().max()) <= 16 * n * 2.0 ** -53 + 1e-14 * float(ref.norm())
