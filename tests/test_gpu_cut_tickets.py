"""The counters with which the CTAs of a cut product or a cut attention group find the last arriver: overlapping launches do not share them, however many
launches lie between, and counters that a launch which gave up left behind do not reach a later one."""
import pytest
import torch

from machx_inference_engine_b200 import _lib
from machx_inference_engine_b200.ops.weights import QuantWeight, WFormat

pytestmark = pytest.mark.gpu


def K():
    from machx_inference_engine_b200.ops import cuda
    return cuda


def calls(seed):
    """Launches whose pieces are cut into different numbers of parts: (product, its result when it runs alone)."""
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda:0").to(torch.bfloat16)
    fns = []
    for M, N, Kd in ((12, 1024, 4096), (5, 6144, 2880), (33, 130, 8192)):
        x, w = rnd(M, Kd), QuantWeight(WFormat.BF16, N, Kd, 1, rnd(1, N, Kd))

        def product(x=x, w=w):
            out = torch.empty(x.shape[0], w.N, dtype=torch.float32, device=x.device)
            K()._gemm_rows(x, w, out, 1, None, None, 0, 0.0, 0.0, x.shape[0])
            return out
        fns.append(product)
    for lens, n_q, n_kv, hd in (([900, 37, 4000], 32, 8, 128), ([5000], 8, 1, 64)):
        nb = -(-max(lens) // 128)
        kc, vc = rnd(len(lens) * nb, n_kv, 128, hd), rnd(len(lens) * nb, n_kv, 128, hd)
        table = torch.arange(len(lens) * nb, dtype=torch.int32, device="cuda:0").view(len(lens), nb)
        a = (rnd(len(lens), n_q, hd), kc, vc, table, torch.tensor(lens, dtype=torch.int32, device="cuda:0"), torch.arange(len(lens) + 1, device="cuda:0").int(), 1)
        fns.append(lambda a=a: K().attention(*a))
    torch.cuda.synchronize()
    want = []
    for f in fns:
        want.append(f())
        torch.cuda.synchronize()
    return fns, want


def captured(fns, n):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = [fns[i % len(fns)]() for i in range(n)]
    return graph, out


def same(out, want):
    return all(torch.equal(o, want[i % len(want)]) for i, o in enumerate(out))


def test_eager_launches_beside_replays_of_a_graph_with_more_launches_than_any_rotation():
    fns, want = calls(1)
    graph, out = captured(fns, 75)
    side, eager = torch.cuda.Stream(), []
    side.wait_stream(torch.cuda.current_stream())
    for r in range(4):
        graph.replay()
        with torch.cuda.stream(side):
            eager = [fns[(i + r) % len(fns)]() for i in range(65 + 5 * r)]
        torch.cuda.synchronize()
        assert same(out, want) and same(eager, [want[(i + r) % len(want)] for i in range(len(want))])


def test_two_graphs_on_two_streams():
    fns, want = calls(2)
    (ga, a), (gb, b) = captured(fns, 70), captured(fns[::-1], 70)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(4):
        ga.replay()
        with torch.cuda.stream(side):
            gb.replay()
    torch.cuda.synchronize()
    assert same(a, want) and same(b, want[::-1])


def test_counters_of_a_launch_that_gave_up_are_dropped_with_its_status(monkeypatch):
    fns, want = calls(3)
    graph, out = captured(fns, 5)
    torch.cuda.synchronize()
    assert K()._stream_tickets and all(int(t.abs().sum()) == 0 for t, *_ in K()._stream_tickets.values())      # every launch leaves its counters at zero
    for t, *_ in K()._stream_tickets.values():                  # as after a launch some of whose warps counted and some did not
        t.fill_(1)
    torch.cuda.synchronize()
    with monkeypatch.context() as m:
        m.setattr(_lib.cuda(), "mx_status_read_and_clear", lambda: 2)
        with pytest.raises(K().KernelError):
            K().check_status()
    assert same([f() for f in fns], want)
    graph.replay()
    torch.cuda.synchronize()
    assert same(out, want)


def test_a_stream_keeps_its_counters_and_shares_them_with_no_other():
    dev, side = torch.device("cuda", 0), torch.cuda.Stream()
    a = K()._tickets(dev)
    with torch.cuda.stream(side):
        b = K()._tickets(dev)
    assert a is K()._tickets(dev) and a[0].data_ptr() != b[0].data_ptr() and len(K()._stream_tickets) <= K().STREAM_TICKETS_MAX
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        c = K()._tickets(dev)
        assert c is K()._tickets(dev)
    assert c[0].data_ptr() not in (a[0].data_ptr(), b[0].data_ptr())
    K()._tickets(dev)
    assert not K()._capture_tickets
