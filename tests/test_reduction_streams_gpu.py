"""One-launch reductions of one context on several streams and from replayed
graphs: their counts of finished blocks are their own, so whatever overlaps, the
results are those of the same calls made one at a time, bit by bit (the
reductions are deterministic), and later calls are not affected.  Captured
reductions of one context share their partials: their replays follow one
another here, beside uncaptured calls on other streams."""
import pytest

pytestmark = pytest.mark.gpu
SIZES = [513, 5000, 70001, 400000, 3000001]


@pytest.fixture()
def own():
    import libgpublas_gb300 as g
    d = g.Device(0)
    yield d
    d.set_stream(None)
    d.close()


class Vectors:
    def __init__(self):
        import torch
        gen = torch.Generator(device="cuda")
        gen.manual_seed(9)
        self.x, self.y = (torch.rand(max(SIZES), dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
                          for _ in range(2))
        torch.cuda.synchronize()

    def new(self):
        import torch
        return (torch.full((2,), float("nan"), dtype=torch.float64, device="cuda"),
                torch.full((2,), -1, dtype=torch.int32, device="cuda"))

    def calls(self, dev, n, out):
        f, i = out
        dev.ddot(n, self.x, 1, self.y, 1, f)
        dev.dnrm2(n, self.x, 1, f[1:])
        dev.idamax(n, self.x, 1, i)
        dev.idamin(n, self.y, 1, i[1:])

    def alone(self, dev):
        """Every size, one call at a time."""
        import torch
        ref = []
        for n in SIZES:
            out = self.new()
            torch.cuda.synchronize()
            self.calls(dev, n, out)
            dev.sync()
            ref.append(out)
        return ref


def same(a, b):
    import torch
    return torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("count", [2, 24])   # fewer and more streams than the context keeps entries for
def test_streams(own, count):
    import torch
    v = Vectors()
    ref = v.alone(own)
    streams = [torch.cuda.Stream() for _ in range(count)]
    outs = [(i % len(SIZES), v.new()) for i in range(240)]
    torch.cuda.synchronize()
    for r, (i, out) in enumerate(outs):
        own.set_stream(streams[r % count].cuda_stream)
        v.calls(own, SIZES[i], out)
    torch.cuda.synchronize()
    for i, out in outs:
        assert same(out, ref[i])
    own.set_stream(None)
    for a, b in zip(v.alone(own), ref):   # nothing is left behind
        assert same(a, b)


def test_replays_beside_other_calls(own):
    import torch
    v = Vectors()
    ref = v.alone(own)
    st, side = torch.cuda.Stream(), torch.cuda.Stream()
    outs = [v.new() for _ in SIZES]
    torch.cuda.synchronize()
    own.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        for n, out in zip(SIZES, outs):
            v.calls(own, n, out)
    own.set_stream(None)
    for _ in range(10):
        for f, i in outs:
            f.fill_(float("nan"))
            i.fill_(-1)
        eager = [(r % len(SIZES), v.new()) for r in range(20)]
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            graph.replay()
        for i, out in eager:
            v.calls(own, SIZES[i], out)
        torch.cuda.synchronize()
        for got, want in zip(outs, ref):
            assert same(got, want)
        for i, out in eager:
            assert same(out, ref[i])


def test_more_captured_calls_than_counters(own):
    """The context has 16384 counters for captured reductions."""
    import torch
    v = Vectors()
    n = SIZES[1]
    ref = v.alone(own)[1]
    st = torch.cuda.Stream()
    f = torch.zeros(16500, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    own.set_stream(st.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        for r in range(16500):
            own.ddot(n, v.x, 1, v.y, 1, f[r:])
    for _ in range(2):
        f.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(f, ref[0][:1].expand(16500))
