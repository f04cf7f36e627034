"""Grouped DGEMM tiles at their edges (rows left out by warp, columns by half
tile, padding of the last 8-k panel), with 32 x 32 and with 64 x 64 tiles, in
every transposition: bit for bit the result of gbx_dgemm.  The tile is set
through the autotuner's cache file, read once per process."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROG = r"""
import itertools, sys
import torch
import libgpublas_gb300 as g
dev = g.Device(0)
gen = torch.Generator(device="cuda"); gen.manual_seed(1)
edges = [1, 2, 3, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 100]
ks = [0, 1, 7, 8, 9, 16, 70]
ops, keep = [], []
for i, (m, n) in enumerate(itertools.product(edges, edges)):
    k, t = ks[i % len(ks)], (i * 7) % 4
    ta, tb = "NT"[t & 1], "NT"[t >> 1]
    u = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
    a = u(*((max(k, 1), m + 1) if ta == "N" else (m, max(k, 1))))
    b = u(*((n, max(k, 1)) if tb == "N" else (max(k, 1), n + 2)))
    c = u(n, m + 3)
    alpha, beta = (1.0, 0.5) if i % 3 else (-0.25, 0.0)
    ref = c.clone()
    keep.append((a, b, c, ref))
    args = (m, n, k, alpha, beta, a.shape[1], b.shape[1], m + 3)
    ops.append(g.GbxOp(kind=1, transa=ta.encode(), transb=tb.encode(), m=m, n=n, k=k, alpha=alpha, beta=beta,
                       A=a.data_ptr(), lda=a.shape[1], B=b.data_ptr(), ldb=b.shape[1], C=c.data_ptr(), ldc=m + 3))
torch.cuda.synchronize()
for o, (a, b, c, ref) in zip(ops, keep):
    assert dev.dgemm(o.transa, o.transb, o.m, o.n, o.k, o.alpha, a, o.lda, b, o.ldb, o.beta, ref, o.ldc) == 0
plan = dev.plan_create(ops)
dev.plan_launch(plan)
dev.sync()
bad = [(o.m, o.n, o.k) for o, (a, b, c, ref) in zip(ops, keep) if not torch.equal(c, ref)]
print("bad", bad)
sys.exit(1 if bad else 0)
"""


@pytest.mark.parametrize("variant", [0, 1])
def test_tiles_equal_dgemm(tmp_path, variant):
    import torch
    cache = tmp_path / "autotune.json"
    cache.write_text(json.dumps({torch.cuda.get_device_name(0) + " trimmed tiles": [variant] * 6}) + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROG], cwd=root, env=dict(os.environ, GBX_AUTOTUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
