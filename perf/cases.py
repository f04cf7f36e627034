"""Performance cases of the BLAS library: what its callers run, through the
public entry points (the gbx_* device ABI, grouped plans and the Fortran
symbols).

Every case is a dict of plain values; `kind` names the code path:

    gemm      gbx_dgemm on device operands
    sgemm     sgemm_ (Fortran ABI) on device-resident operands
    host      dgemm_ (Fortran ABI) on ordinary host memory, copies included
    ozaki     gbx_dgemm_ozaki, the split-precision product at its default
              tolerance
    trsm      gbx_dtrsm with many right-hand sides
    cholesky  one caller's blocked Cholesky: dpotrf of the diagonal block,
              dtrsm of the panel, dsyrk + dgemm of the trailing matrix
              (FP64 or Ozaki forms)
    batched   many small uneven DGEMM / DTRSM calls as one grouped plan,
              replayed from its CUDA graph
    reflect   a Householder reflector applied from the left and from the
              right (DGEMV T + DGER, DGEMV N + DGER), the inner step of a
              bidiagonalisation
    pcg       the matrix work of one preconditioned CG iteration: DSYMV and
              a forward and a backward DTRSV
    vectors   the vector work of one CG iteration: DDOT, two DAXPYs, DNRM2,
              IDAMAX
"""
import math

import numpy as np
import torch

import libgpublas_gb300 as g

_device = None


def _dev():
    """The library context that a program creates once and keeps."""
    global _device
    if _device is None:
        _device = g.Device(0)
    return _device


def _on_stream():
    """torch work ordered with the library's calls (its stream is its own)."""
    return torch.cuda.stream(torch.cuda.ExternalStream(_dev().stream()))


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a latency-bound small product: what a program that makes many tiny
        # calls waits for
        {"name": "dgemm_64", "kind": "gemm", "ta": "N", "tb": "N", "m": 64, "n": 64, "k": 64, "pad": 0, "beta": 1.0},
        # the FP64 workhorse at an ordinary large, ragged size, transposed,
        # with a leading dimension that is not the row count
        {"name": "dgemm_tn_ragged", "kind": "gemm", "ta": "T", "tb": "N", "m": 2999, "n": 2500, "k": 2777, "pad": 5,
         "beta": 0.5},
        # single precision at the usual benchmark size
        {"name": "sgemm_4096", "kind": "sgemm", "ta": "N", "tb": "N", "m": 4096, "n": 4096, "k": 4096, "beta": 0.5},
        # an unmodified Fortran program's dgemm_ on its own memory
        {"name": "dgemm_host_512", "kind": "host", "ta": "N", "tb": "N", "m": 512, "n": 512, "k": 512, "beta": 0.5},
        # the opt-in split-precision product, entries over 2^-8 .. 2^8
        {"name": "ozaki_8192", "kind": "ozaki", "ta": "N", "tb": "N", "m": 8192, "n": 8192, "k": 8192, "spread": 8,
         "beta": 0.0},
        # a large triangular solve with many right-hand sides
        {"name": "dtrsm_8192", "kind": "trsm", "side": "L", "uplo": "L", "ta": "N", "diag": "N", "order": 8192,
         "rhs": 1024, "pad": 0},
        # one caller of the serving trace, in the Ozaki forms
        {"name": "cholesky_4096", "kind": "cholesky", "n": 4096, "nb": 256, "ozaki": True},
        # the batched workload at a fifth of its size
        {"name": "batched_5000", "kind": "batched", "gemms": 4000, "trsms": 1000},
        # Householder bidiagonalisation, early step (matrix larger than L2)
        {"name": "reflect_8192", "kind": "reflect", "m": 8192, "n": 8192, "pad": 0},
        # dense preconditioned CG
        {"name": "pcg_8192", "kind": "pcg", "n": 8192, "uplo": "L"},
        # CG vectors much larger than L2, and small enough that the calls'
        # latency is all there is
        {"name": "vectors_64m", "kind": "vectors", "n": 1 << 26, "inc": 1},
        {"name": "vectors_10k", "kind": "vectors", "n": 10001, "inc": 1},
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "sgemm", "host", "ozaki", "trsm", "cholesky", "batched", "reflect", "pcg", "vectors"])
    c = {"kind": kind}
    if kind in ("gemm", "sgemm", "host", "ozaki"):
        lo, hi = {"gemm": (48, 3000), "sgemm": (48, 6000), "host": (64, 900), "ozaki": (512, 8192)}[kind]
        c.update(ta=rng.choice("NT"), tb=rng.choice("NT"), m=_loguni(rng, lo, hi), n=_loguni(rng, lo, hi),
                 k=_loguni(rng, lo, hi), beta=rng.choice([0.0, 0.5, 1.0]))
        if kind == "gemm":
            c["pad"] = rng.choice([0, 0, 1, 6])
        if kind == "ozaki":
            c["spread"] = rng.choice([0, 8, 24])
    elif kind == "trsm":
        c.update(side=rng.choice("LR"), uplo=rng.choice("LU"), ta=rng.choice("NT"), diag=rng.choice("NU"),
                 order=_loguni(rng, 100, 8000), rhs=_loguni(rng, 16, 1000), pad=rng.choice([0, 0, 3]))
    elif kind == "cholesky":
        c.update(n=_loguni(rng, 500, 4000), nb=rng.choice([128, 256]), ozaki=rng.random() < 0.5)
    elif kind == "batched":
        count = _loguni(rng, 200, 4800)
        c.update(gemms=count - count // 5, trsms=count // 5)
    elif kind == "reflect":
        c.update(m=_loguni(rng, 200, 9000), n=_loguni(rng, 200, 7000), pad=rng.choice([0, 0, 1, 4]))
    elif kind == "pcg":
        c.update(n=_loguni(rng, 200, 9000), uplo=rng.choice("LU"))
    else:
        inc = rng.choice([1, 1, 1, 2])
        c.update(n=_loguni(rng, 500, (1 << 26) // inc), inc=inc)
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _uni(gen, *shape, dtype=torch.float64):
    """uniform[-1, 1]"""
    return torch.rand(*shape, dtype=dtype, device="cuda", generator=gen).mul_(2.0).sub_(1.0)


def _triangle(gen, n, ld=None):
    """A triangle's square: diagonal uniform[1,2], the rest uniform[-1,1]/n."""
    a = _uni(gen, n, ld or n)
    a.mul_(1.0 / n)
    a.diagonal().copy_(torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).add_(1.0))
    return a


class _Plan:
    """A grouped plan and its operands; given back with the state."""

    def __init__(self, ops):
        self.handle = _dev().plan_create(ops)

    def __del__(self):
        _dev().plan_destroy(self.handle)


def _batched_ops(case, base):
    """(ops, doubles, doubles of right-hand sides): four DGEMMs, then one
    DTRSM, operands packed in one buffer at `base`: all right-hand sides
    first, then the rest.  The sizes follow from the case alone."""
    rng = np.random.default_rng(case["gemms"])

    def loguni(lo, hi, shape):
        return np.rint(np.exp(rng.uniform(math.log(lo), math.log(hi), shape))).astype(int)

    mnk = loguni(8, 512, (case["gemms"], 3))
    orders = loguni(8, 256, case["trsms"])
    rhs = int(16 * orders.sum())
    ops, off, roff = [], rhs + rhs % 2, 0
    gi = ti = 0
    while gi < len(mnk) or ti < len(orders):
        for m, n, k in mnk[gi:gi + 4].tolist():
            pa, pb, pc = base + 8 * off, base + 8 * (off + m * k), base + 8 * (off + m * k + k * n)
            ops.append(g.GbxOp(kind=1, transa=b"N", transb=b"N", m=m, n=n, k=k, alpha=1.0, beta=0.5, A=pa, lda=m,
                               B=pb, ldb=k, C=pc, ldc=m))
            off += m * k + k * n + m * n
        gi += 4
        if ti < len(orders):
            o = int(orders[ti])
            ops.append(g.GbxOp(kind=2, transa=b"N", side=b"L", uplo=b"L", diag=b"N", m=o, n=16, alpha=1.0,
                               A=base + 8 * off, lda=o, C=base + 8 * roff, ldc=o))
            off += o * o
            roff += 16 * o
            ti += 1
    return ops, off, rhs


def _cholesky_ops(n, nb, base, info, ozaki):
    """The call list of one caller of the serving trace (column-major, ld n)."""
    gemm, syrk, trsm = (7, 8, 9) if ozaki else (1, 3, 2)
    at = lambda i, j: base + 8 * (j * n + i)   # noqa: E731
    ops = []
    for k in range(0, n, nb):
        kb = min(nb, n - k)
        ops.append(g.GbxOp(kind=6, uplo=b"L", n=kb, B=info, C=at(k, k), ldc=n))
        rest = n - k - kb
        if rest <= 0:
            continue
        ops.append(g.GbxOp(kind=trsm, side=b"R", uplo=b"L", transa=b"T", diag=b"N", m=rest, n=kb, alpha=1.0,
                           A=at(k, k), lda=n, C=at(k + kb, k), ldc=n))
        for j in range(k + kb, n, nb):
            jb = min(nb, n - j)
            ops.append(g.GbxOp(kind=syrk, uplo=b"L", transa=b"N", n=jb, k=kb, alpha=-1.0, beta=1.0, A=at(j, k),
                               lda=n, C=at(j, j), ldc=n))
            below = n - j - jb
            if below > 0:
                ops.append(g.GbxOp(kind=gemm, transa=b"N", transb=b"T", m=below, n=jb, k=kb, alpha=-1.0, beta=1.0,
                                   A=at(j + jb, k), lda=n, B=at(j, k), ldb=n, C=at(j + jb, j), ldc=n))
    return ops


def _inputs(case, seed):
    """The inputs as tensors: a column-major matrix of ld rows and c columns
    is a (c, ld) tensor."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, s = case["kind"], {}
    if kind in ("gemm", "sgemm", "host", "ozaki"):
        m, n, k, pad = case["m"], case["n"], case["k"], case.get("pad", 0)
        ash = (k, m + pad) if case["ta"] == "N" else (m, k + pad)
        bsh = (n, k + pad) if case["tb"] == "N" else (k, n + pad)
        dt = torch.float32 if kind == "sgemm" else torch.float64
        for name, shape in (("a", ash), ("b", bsh), ("c", (n, m + pad))):
            s[name] = _uni(gen, *shape, dtype=dt)
            if case.get("spread") and name != "c":
                e = torch.randint(-case["spread"], case["spread"] + 1, shape, device="cuda", generator=gen)
                s[name] = torch.ldexp(s[name], e)
                del e
    elif kind == "trsm":
        o, r, pad = case["order"], case["rhs"], case["pad"]
        s["a"] = _triangle(gen, o, o + pad)
        s["b0"] = _uni(gen, *((r, o + pad) if case["side"] == "L" else (o, r + pad)))
    elif kind == "cholesky":
        n = case["n"]
        w = _uni(gen, n, n)
        s["a0"] = w @ w.T
        s["a0"].diagonal().add_(float(n))
    elif kind == "reflect":
        m, n, pad = case["m"], case["n"], case["pad"]
        s["a"] = _uni(gen, n, m + pad)
        s["v"], s["u"] = _uni(gen, m), _uni(gen, n)
    elif kind == "pcg":
        n = case["n"]
        s["a"], s["l"] = _uni(gen, n, n), _triangle(gen, n)
        s["p"], s["r"] = _uni(gen, n), _uni(gen, n)
    elif kind == "vectors":
        n = case["n"] * case["inc"]
        for name in "xprqz":
            s[name] = _uni(gen, n)
        s["z"].mul_(0.25).add_(s["r"])
    return s


def _fill_batched(case, seed):
    """(flat buffer, ops, doubles of right-hand sides)."""
    ops, total, rhs = _batched_ops(case, 0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    buf = _uni(gen, total)
    for o in ops:   # the triangles: diagonal uniform[1,2], the rest over the order
        if o.kind == 2:
            t = buf[o.A // 8 if o.A else 0:][:o.m * o.m].view(o.m, o.m)
            d = t.diagonal().abs().add_(1.0)
            t.mul_(1.0 / o.m)
            t.diagonal().copy_(d)
    return buf, ops, rhs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batched":
        buf, ops, rhs = _fill_batched(case, seed)
        base = buf.data_ptr()
        for o in ops:
            o.A, o.C = (o.A or 0) + base, (o.C or 0) + base
            if o.kind == 1:
                o.B = o.B + base
        torch.cuda.synchronize()
        s = {"buf": buf, "rhs": rhs, "b0": buf[:rhs].clone(), "plan": _Plan(ops)}
    else:
        s = _inputs(case, seed)
    if kind == "host":
        s = {k: v.cpu().numpy() for k, v in s.items()}
        s["f77"] = g.F77()
    elif kind == "sgemm":
        s["f77"] = g.F77()
    elif kind == "trsm":
        s["x"] = s["b0"].clone()
    elif kind == "cholesky":
        s["x"], s["info"] = s["a0"].clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
        ops = _cholesky_ops(case["n"], case["nb"], s["x"].data_ptr(), s["info"].data_ptr(), case["ozaki"])
        s["ops"], s["count"] = (g.GbxOp * len(ops))(*ops), len(ops)
    elif kind == "reflect":
        s["tau_v"], s["tau_u"] = (2.0 / float(s[k] @ s[k]) for k in "vu")
        s["wt"], s["wn"] = torch.empty_like(s["u"]), torch.empty_like(s["v"])
    elif kind == "pcg":
        s["q"], s["w"] = torch.empty_like(s["p"]), torch.empty_like(s["r"])
    elif kind == "vectors":
        s["rho"], s["nrm"] = (torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(2))
        s["imax"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    s["case"] = dict(case)
    _dev()
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    s, c, dev = state, state["case"], _dev()
    kind = c["kind"]
    if kind == "gemm":
        _, lda = s["a"].shape
        dev.dgemm_checked(c["ta"], c["tb"], c["m"], c["n"], c["k"], 1.0, s["a"], lda, s["b"], s["b"].shape[1],
                          c["beta"], s["c"], s["c"].shape[1])
        return s["c"]
    if kind == "sgemm":
        s["f77"].gemm("s", c["ta"], c["tb"], c["m"], c["n"], c["k"], 1.0, s["a"].data_ptr(), s["a"].shape[1],
                      s["b"].data_ptr(), s["b"].shape[1], c["beta"], s["c"].data_ptr(), s["c"].shape[1])
        return s["c"]
    if kind == "host":
        s["f77"].dgemm(c["ta"], c["tb"], c["m"], c["n"], c["k"], 1.0, s["a"], s["a"].shape[1], s["b"],
                       s["b"].shape[1], c["beta"], s["c"], s["c"].shape[1])
        return s["c"]
    if kind == "ozaki":
        dev.dgemm_ozaki(c["ta"], c["tb"], c["m"], c["n"], c["k"], 1.0, s["a"], s["a"].shape[1], s["b"],
                        s["b"].shape[1], c["beta"], s["c"], s["c"].shape[1], want_slices=False)
        return s["c"]
    if kind == "trsm":
        with _on_stream():   # the solve is in place: new right-hand sides
            s["x"].copy_(s["b0"])
        m, n = (c["order"], c["rhs"]) if c["side"] == "L" else (c["rhs"], c["order"])
        dev.dtrsm(c["side"], c["uplo"], c["ta"], c["diag"], m, n, 1.0, s["a"], s["a"].shape[1], s["x"],
                  s["x"].shape[1])
        return s["x"]
    if kind == "cholesky":
        with _on_stream():   # the factorisation is in place: a new matrix
            s["x"].copy_(s["a0"])
        dev.ops_run(s["ops"], s["count"])
        return [s["x"], s["info"]]
    if kind == "batched":
        with _on_stream():
            s["buf"][:s["rhs"]].copy_(s["b0"])
        dev.plan_launch(s["plan"].handle, graph=True)
        return s["buf"]
    if kind == "reflect":
        m, n, ld = c["m"], c["n"], s["a"].shape[1]
        dev.dgemv("T", m, n, 1.0, s["a"], ld, s["v"], 1, 0.0, s["wt"], 1)
        L, ctx = dev.L, dev.ctx
        _ok(L.gbx_dger(ctx, m, n, -s["tau_v"], s["v"].data_ptr(), 1, s["wt"].data_ptr(), 1, s["a"].data_ptr(), ld))
        dev.dgemv("N", m, n, 1.0, s["a"], ld, s["u"], 1, 0.0, s["wn"], 1)
        _ok(L.gbx_dger(ctx, m, n, -s["tau_u"], s["wn"].data_ptr(), 1, s["u"].data_ptr(), 1, s["a"].data_ptr(), ld))
        return [s["a"], s["wt"], s["wn"]]
    if kind == "pcg":
        n, up = c["n"], c["uplo"].encode()
        with _on_stream():
            s["w"].copy_(s["r"])
        L, ctx = dev.L, dev.ctx
        _ok(L.gbx_dsymv(ctx, up, n, 1.0, s["a"].data_ptr(), n, s["p"].data_ptr(), 1, 0.0, s["q"].data_ptr(), 1))
        # M = L L^T, or U^T U
        for tr in (b"NT" if c["uplo"] == "L" else b"TN"):
            _ok(L.gbx_dtrsv(ctx, up, bytes([tr]), b"N", n, s["l"].data_ptr(), n, s["w"].data_ptr(), 1))
        return [s["q"], s["w"]]
    n, inc = c["n"], c["inc"]
    dev.ddot(n, s["r"], inc, s["z"], inc, s["rho"])
    dev.daxpy(n, 1e-3, s["p"], inc, s["x"], inc)
    dev.daxpy(n, -1e-3, s["q"], inc, s["r"], inc)
    dev.dnrm2(n, s["r"], inc, s["nrm"])
    dev.idamax(n, s["r"], inc, s["imax"])
    return [s["x"], s["r"], s["rho"], s["nrm"], s["imax"]]


def _ok(status):
    if status != 0:
        raise g.GbxError(f"status {status}")


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("gemm", "sgemm", "host", "ozaki"):
        m, n, k = case["m"], case["n"], case["k"]
        e = 4 if kind == "sgemm" else 8
        return {"bytes": e * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2.0 * m * n * k}
    if kind == "trsm":
        o, r = case["order"], case["rhs"]
        return {"bytes": 8 * (o * (o + 1) // 2 + 2 * o * r), "flops": float(o) * o * r}
    if kind == "cholesky":
        n = case["n"]
        return {"bytes": 8 * n * (n + 1), "flops": n ** 3 / 3.0}
    if kind == "batched":
        ops, _, _ = _batched_ops(case, 0)
        b = sum(8 * (o.m * o.k + o.k * o.n + 2 * o.m * o.n) if o.kind == 1 else 4 * o.m * (o.m + 1) + 256 * o.m
                for o in ops)
        f = sum(2.0 * o.m * o.n * o.k if o.kind == 1 else 16.0 * o.m * o.m for o in ops)
        return {"bytes": b, "flops": f}
    if kind == "reflect":   # each side: the product reads the matrix, the update reads and writes it
        return {"bytes": 48 * case["m"] * case["n"], "flops": 8.0 * case["m"] * case["n"]}
    if kind == "pcg":       # one triangle each for DSYMV and the two solves
        n = case["n"]
        return {"bytes": 12 * n * (n + 1) + 48 * n, "flops": 4.0 * n * n}
    return {"bytes": 80 * case["n"], "flops": 8.0 * case["n"]}


# --------------------------------------------------------------------------
# the same in plain 64-bit torch
# --------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "batched":
        buf, ops, _ = _fill_batched(case, seed)
        for o in ops:
            part = lambda p, r, q: buf[(p or 0) // 8:][:r * q].view(q, r)   # noqa: E731  (column-major r x q)
            if o.kind == 1:
                cm = part(o.C, o.m, o.n)
                cm.copy_(0.5 * cm + part(o.B, o.k, o.n) @ part(o.A, o.m, o.k))
            else:
                x = part(o.C, o.m, 16)
                x.copy_(torch.linalg.solve_triangular(part(o.A, o.m, o.m).T, x.T, upper=False).T)
        return buf
    s = _inputs(case, seed)
    if kind in ("gemm", "sgemm", "host", "ozaki"):
        m, n, k = case["m"], case["n"], case["k"]
        a = s["a"][:, :m].T if case["ta"] == "N" else s["a"][:, :k]   # op(A), m x k
        b = s["b"][:, :k].T if case["tb"] == "N" else s["b"][:, :n]   # op(B), k x n
        out = s["c"].double()
        out[:, :m] = case["beta"] * out[:, :m] + (a.double() @ b.double()).T
        return out.cpu().numpy() if kind == "host" else out
    if kind == "trsm":
        o, r = case["order"], case["rhs"]
        t = s["a"][:, :o].T   # the stored matrix
        lower = case["uplo"] == "L"
        t = t.tril() if lower else t.triu()
        if case["ta"] == "T":
            t, lower = t.T, not lower
        x = s["b0"]
        left = case["side"] == "L"
        rows = o if left else r
        b = x[:, :rows].T
        x[:, :rows] = torch.linalg.solve_triangular(t, b, upper=not lower, left=left,
                                                    unitriangular=case["diag"] == "U").T
        return x
    if kind == "cholesky":
        # lower triangle (column-major): the upper triangle of the row-major tensor
        low = torch.linalg.cholesky(s["a0"])
        return [s["a0"].tril(-1) + low.T, None]
    if kind == "reflect":
        m, a, v, u = case["m"], s["a"], s["v"], s["u"]
        am = a[:, :m].T
        wt = am.T @ v
        am -= torch.outer((2.0 / (v @ v)) * v, wt)
        wn = am @ u
        am -= torch.outer((2.0 / (u @ u)) * wn, u)
        return [a, wt, wn]
    if kind == "pcg":
        a = s["a"].T   # column-major storage
        sym = a.tril() + a.tril(-1).T if case["uplo"] == "L" else a.triu() + a.triu(1).T
        low = s["l"].T.tril() if case["uplo"] == "L" else s["l"].T.triu().T   # U^T U
        z = torch.linalg.solve_triangular(low, s["r"][:, None], upper=False)
        z = torch.linalg.solve_triangular(low.T, z, upper=True)
        return [sym @ s["p"], z[:, 0]]
    inc = case["inc"]
    x, p, r, q, z = (s[k][::inc] for k in "xprqz")
    rho = (r * z).sum().reshape(1)
    x += 1e-3 * p
    r -= 1e-3 * q
    return [s["x"], s["r"], rho, r.norm().reshape(1), None]
