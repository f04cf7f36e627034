"""SGEMM calls of one context on several streams, and captured ones, are
independent of one another: every call has scratch of its own, and a capture
uses none.  Results are compared bit by bit with those of the same call made
alone (captured: made by another capture), so there is no tolerance."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def make(seed, m, n, k):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    a, b, c = (torch.rand(r, s, device="cuda", generator=gen) * 2 - 1 for r, s in ((k, m), (n, k), (n, m)))
    return {"a": a, "b": b, "c": c, "size": (m, n, k)}


def sgemm(dev, p, out):
    m, n, k = p["size"]
    assert dev.L.gbx_sgemm(dev.ctx, b"N", b"N", m, n, k, C.c_float(1.0), C.c_void_p(p["a"].data_ptr()), m,
                           C.c_void_p(p["b"].data_ptr()), k, C.c_float(0.0), C.c_void_p(out.data_ptr()), m) == 0


def alone(dev, p):
    import torch
    out = torch.empty_like(p["c"])
    torch.cuda.synchronize()
    sgemm(dev, p, out)
    dev.sync()
    return out


def capture(dev, p, out):
    import torch
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    dev.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        sgemm(dev, p, out)
    dev.set_stream(None)
    return graph


@pytest.fixture()
def own():
    import libgpublas_gb300 as g
    d = g.Device(0)
    yield d
    d.set_stream(None)
    d.close()


def test_one_context_on_two_streams(own):
    import torch
    probs = [make(i, 1500 + 100 * i, 1400, 1300) for i in range(4)]
    ref = [alone(own, p) for p in probs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.empty_like(p["c"]) for p in probs] for _ in range(5)]
    torch.cuda.synchronize()
    for row in outs:
        for i, p in enumerate(probs):
            own.set_stream(streams[i % 2].cuda_stream)
            sgemm(own, p, row[i])
    torch.cuda.synchronize()
    for row in outs:
        for i in range(len(probs)):
            assert torch.equal(row[i], ref[i])


def test_more_streams_than_blocks_of_scratch(own):
    """Six streams and products of growing size: blocks are waited for and replaced."""
    import torch
    probs = [make(40 + i, 600 + 150 * i, 700, 900) for i in range(6)]
    ref = [alone(own, p) for p in probs]
    streams = [torch.cuda.Stream() for _ in range(6)]
    outs = [[torch.empty_like(p["c"]) for p in probs] for _ in range(4)]
    torch.cuda.synchronize()
    for r, row in enumerate(outs):
        for i, p in enumerate(probs):
            own.set_stream(streams[(i + r) % 6].cuda_stream)
            sgemm(own, p, row[i])
    torch.cuda.synchronize()
    for row in outs:
        for i in range(len(probs)):
            assert torch.equal(row[i], ref[i])


def test_two_contexts_in_turn(own):
    import torch
    import libgpublas_gb300 as g
    other = g.Device(0)
    probs = [make(10 + i, 900, 800 + 64 * i, 1100) for i in range(2)]
    ref = [alone(own, p) for p in probs]
    outs = [[torch.empty_like(p["c"]) for p in probs] for _ in range(10)]
    torch.cuda.synchronize()
    for row in outs:
        for d, p, o in ((own, probs[0], row[0]), (other, probs[1], row[1])):
            sgemm(d, p, o)
    torch.cuda.synchronize()
    other.close()
    for row in outs:
        for i in range(2):
            assert torch.equal(row[i], ref[i])


def test_replay_after_a_larger_call_and_beside_others(own):
    import torch
    p, big = make(20, 700, 700, 600), make(21, 3000, 2900, 2800)
    alone(own, p)   # the context has run this product before
    want, got = torch.empty_like(p["c"]), torch.empty_like(p["c"])
    first = capture(own, p, want)
    first.replay()
    torch.cuda.synchronize()
    graph = capture(own, p, got)
    ref = alone(own, big)
    side = torch.cuda.Stream()
    out = torch.empty_like(big["c"])
    for _ in range(3):
        got.fill_(float("nan"))
        torch.cuda.synchronize()
        sgemm(own, big, out)
        with torch.cuda.stream(side):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(out, ref)


@pytest.mark.parametrize("value", [float("inf"), 1e-25])
def test_replays_do_not_depend_on_earlier_operands(own, value):
    """An operand that the split does not cover leaves no trace."""
    import torch
    p = make(30, 800, 700, 600)
    out = torch.empty_like(p["c"])
    graph = capture(own, p, out)
    graph.replay()
    torch.cuda.synchronize()
    want, plain = out.clone(), alone(own, p)
    keep = float(p["a"][3, 5])
    p["a"][3, 5] = value
    graph.replay()
    alone(own, p)
    p["a"][3, 5] = keep
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert torch.equal(alone(own, p), plain)
