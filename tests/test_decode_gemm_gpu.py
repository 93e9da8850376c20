"""The weight-streaming decode GEMM against fp32, where its three ways to cut the work meet their edges."""
import pytest
import torch

from gcore_b200.ops import _lib
from gcore_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


# (N, K): one piece per CTA with equal and unequal pieces, ragged tiles and k-blocks, runs that divide tiles, runs of whole
# tiles, one tile more than SMs; more than half as many tiles as SMs, whole and divided
SHAPES = [(3584, 3584), (4608, 1600), (700, 9000), (7168, 1152), (24576, 512), (32768, 520), (19072, 712), (300, 20000),
          (9600, 1024), (9728, 2560), (13000, 416)]


@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("T", [1, 16, 17, 63, 128])
def test_stream_gemm(N, K, T):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N + K + T)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device="cuda")
    ref = x.double() @ w.double().t()
    before = G.LAUNCHES["gemm"]
    y = G.linear_forward(x, w, out_dtype=torch.float32)
    assert N * K >= 5 << 20 and G.LAUNCHES["gemm"] == before + 1
    # fp32 sums of K products of exact bf16 values: sqrt(K) roundings of 2^-24 relative to the sum of magnitudes
    bound = 4 * K ** 0.5 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert ((y.double() - ref).abs() <= bound + 1e-12).all()
    yb = G.linear_forward(x, w, b.bfloat16())
    refb = ref + b.bfloat16().double()
    assert ((yb.double() - refb).abs() <= refb.abs() * 2.0 ** -8 + bound + 1e-12).all()
    out = torch.full((T, N + 24), 7.0, device="cuda", dtype=torch.float32)[:, 8:N + 8]     # strided result
    G.linear_forward(x, w, b, out=out)
    assert torch.equal(out, G.linear_forward(x, w, b, out_dtype=torch.float32))
    assert bool((out._base[:, :8] == 7).all()) and bool((out._base[:, N + 8:] == 7).all())
    _lib.check_device_errors()


def test_streams_and_captured_branches_keep_their_counters_apart():
    """Launches that may overlap: four streams at once, and two branches of one graph."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    T, N, K = 8, 4608, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn(T, K, generator=g, device="cuda").bfloat16() for _ in range(4)]
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = [G.linear_forward(x, w, out_dtype=torch.float32) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    outs = [[] for _ in xs]
    for _ in range(20):
        for s, x, o in zip(streams, xs, outs):
            with torch.cuda.stream(s):
                o.append(G.linear_forward(x, w, out_dtype=torch.float32))
    torch.cuda.synchronize()
    assert all(torch.equal(y, r) for o, r in zip(outs, ref) for y in o)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        side.wait_stream(torch.cuda.current_stream())
        a = G.linear_forward(xs[0], w, out_dtype=torch.float32)
        with torch.cuda.stream(side):
            b = G.linear_forward(xs[1], w, out_dtype=torch.float32)
        torch.cuda.current_stream().wait_stream(side)
    for _ in range(5):
        a.zero_()
        b.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(a, ref[0]) and torch.equal(b, ref[1])
    _lib.check_device_errors()


@pytest.mark.parametrize("N,K", [(3584, 4096), (1024, 512)])
def test_refuses_a_weight_of_another_width(N, K):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    w = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="contraction mismatch"):
        G.linear_forward(w[:4, :K - 64].contiguous(), w)


def _problem(seed, n=2):
    T, N, K = 8, 4608, 4096
    g = torch.Generator(device="cuda").manual_seed(seed)
    xs = [torch.randn(T, K, generator=g, device="cuda").bfloat16() for _ in range(n)]
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    return xs, w, [G.linear_forward(x, w, out_dtype=torch.float32) for x in xs]


def test_no_two_live_graphs_share_counters(monkeypatch):
    """More captures than a fixed table would hold; the first and the last graph at once on two streams."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    xs, w, ref = _problem(5)
    own, seen = G._counters, []
    monkeypatch.setattr(G, "_counters", lambda *a: (lambda c: (seen.append(c.data_ptr()), c)[1])(own(*a)))
    graphs, outs = [], []
    for i in range(132):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs.append([G.linear_forward(xs[i % 2], w, out_dtype=torch.float32) for _ in range(2)])
        graphs.append(graph)
    assert len(seen) == 264 and len(set(seen)) == 132       # one for both products of a capture
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(50):
        for s, graph in zip(streams, (graphs[0], graphs[-1])):
            with torch.cuda.stream(s):
                graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(y, ref[0]) for y in outs[0]) and all(torch.equal(y, ref[1]) for y in outs[-1])
    G.linear_forward(xs[0], w)
    assert not G._CAPTURED                                   # nothing keeps a finished capture's memory
    _lib.check_device_errors()


def test_first_use_in_a_capture_and_in_two_threads(monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import threading
    xs, w, ref = _problem(6)
    G._COUNTERS.clear()
    graph = torch.cuda.CUDAGraph()
    before = G.LAUNCHES["gemm"]
    with torch.cuda.graph(graph):
        y = G.linear_forward(xs[0], w, out_dtype=torch.float32)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref[0]) and G.LAUNCHES["gemm"] == before + 1   # the same kernel as outside
    monkeypatch.setattr(G, "COUNTER_OWNERS", 1)              # owners push one another out all the time
    outs, go = [[], []], threading.Barrier(2)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            go.wait()
            for _ in range(100):
                outs[i].append(G.linear_forward(xs[i], w, out_dtype=torch.float32))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert all(len(o) == 100 and all(torch.equal(y, r) for y in o) for o, r in zip(outs, ref))
    _lib.check_device_errors()


def test_counters_start_over_after_a_reported_error():
    """What a launch that gave up leaves behind: counters that are not zero, on every stream and inside a graph."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    xs, w, ref = _problem(7)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = G.linear_forward(xs[1], w, out_dtype=torch.float32)
        captured = list(G._CAPTURED.values())
    for c in list(G._COUNTERS.values()) + captured:
        c.fill_(3)
    torch.cuda.synchronize()
    _lib.err_flag(w.device).fill_(1)
    with pytest.raises(RuntimeError, match="timed-out wait"):
        _lib.check_device_errors()
    for _ in range(3):
        graph.replay()
        assert torch.equal(y, ref[1]) and torch.equal(G.linear_forward(xs[0], w, out_dtype=torch.float32), ref[0])
    _lib.check_device_errors()


@pytest.mark.parametrize("N,K", [(4608, 3584), (24576, 512), (32768, 520)])
def test_ends_while_an_earlier_error_stands(N, K):
    """Another kernel's error makes waits give up early: the launch ends, and the one after the report is right."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(8, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = G.linear_forward(x, w, out_dtype=torch.float32)
    for _ in range(5):
        _lib.err_flag(w.device).fill_(1)
        G.linear_forward(x, w)
        with pytest.raises(RuntimeError, match="timed-out wait"):
            _lib.check_device_errors()
        assert torch.equal(G.linear_forward(x, w, out_dtype=torch.float32), ref)
    _lib.check_device_errors()


# few feature tiles: one piece per CTA; 4 to 48 pieces a tile, ragged ones among them
@pytest.mark.parametrize("N,K", [(4608, 1600), (2048, 4096), (700, 9000), (300, 20000)])
@pytest.mark.parametrize("T", [1, 17, 128])
def test_shares_left_to_the_last_piece(N, K, T, monkeypatch):
    """Without patience every CTA but the one that brings a tile's last piece leaves its share to that one."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N + K + T)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = G.linear_forward(x, w, out_dtype=torch.float32)
    monkeypatch.setattr(G, "SHARE_WAIT", 0)
    for _ in range(20):                                      # on the same counters, which have to be back at zero
        assert torch.equal(G.linear_forward(x, w, out_dtype=torch.float32), ref)
    torch.cuda.synchronize()
    assert all(not c.any() for c in G._COUNTERS.values())
    _lib.check_device_errors()
