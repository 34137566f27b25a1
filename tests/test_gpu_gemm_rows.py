"""Weight-streaming products of a few rows (csrc/cuda/gemm_rows.cu) against fp64.

Bound: the operands are exact (bf16, or int8 codes and fp16 scales), the sums fp32.  Rounding to bf16 moves an element, and so the 2-norm, by at most
2^-8 = 3.9e-3; fp32 results differ by the order of the sums, about 1e-6, and by what the tensor cores cut off:
up to a unit in the last place of the running sum (2^-23) at each of the K / 16 additions, half of it on average."""
import pytest
import torch

from machx_inference_engine_b200 import ops
from machx_inference_engine_b200.ops.weights import QuantWeight, WFormat, from_dense

pytestmark = pytest.mark.gpu


def K():
    from machx_inference_engine_b200.ops import cuda
    return cuda


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def weight(fmt, N, Kd, E=1, seed=0):
    g = torch.Generator().manual_seed(seed)
    return from_dense(torch.randn(E, N, Kd, generator=g) * 0.05, fmt).to("cuda:0")


def values(w):
    if w.fmt == WFormat.BF16:
        return w.p0.double().reshape(w.E, w.N, w.K)
    d = w.p1.double().reshape(w.E, w.N, -1)[..., :w.K // 32].repeat_interleave(32, dim=-1)
    return w.p0.double().reshape(w.E, w.N, w.K) * d


def product(x, w, out_f32, **kw):
    out = torch.empty(x.shape[0], w.N // 2 if ops.act_gated(kw.get("act", 0)) else w.N, dtype=torch.float32 if out_f32 else torch.bfloat16, device=x.device)
    K()._gemm_rows(x, w, out, 1 if out_f32 else 0, kw.get("bias"), kw.get("row_scale"), kw.get("act", 0), 1.702, 7.0, x.shape[0])
    return out


@pytest.mark.parametrize("fmt", [WFormat.BF16, WFormat.Q8])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 24, 31, 40, 41, 48, 49, 64])
@pytest.mark.parametrize("N,Kd", [(128, 128), (96, 96), (257, 2880), (1000, 4096), (6144, 160), (32, 14336)])
def test_rows_and_ragged_weights(fmt, M, N, Kd):
    x = torch.randn(M, Kd, device="cuda:0").to(torch.bfloat16)
    w = weight(fmt, N, Kd)
    want = x.double() @ values(w)[0].T
    tol = 3e-6 + Kd / 16 * 2.0 ** -24
    assert rel(product(x, w, True), want) < tol
    got = product(x, w, False)
    assert rel(got, want) < 2.0 ** -8
    assert torch.equal(got, product(x, w, False))                    # the parts of a cut tile are added in a fixed order
    bias, rs = torch.randn(N, device=x.device), torch.rand(M, device=x.device)
    assert rel(product(x, w, True, bias=bias, row_scale=rs), (want + bias.double()) * rs.double()[:, None]) < tol


@pytest.mark.parametrize("fmt", [WFormat.BF16, WFormat.Q8])
@pytest.mark.parametrize("act", [ops.ACT_SWIGLU, ops.ACT_SWIGLU_OAI, ops.ACT_GEGLU, ops.ACT_RELU2])
def test_activations(fmt, act):
    from machx_inference_engine_b200.ops import ref
    x = torch.randn(19, 1088, device="cuda:0").to(torch.bfloat16)
    w = weight(fmt, 544, 1088)
    got, want = ops.linear(x, w, act=act, out_f32=True), ref.linear(x.cpu(), w.to("cpu"), act=act, out_f32=True)
    assert rel(got.cpu(), want) < 5e-3                               # (the oracle's Q8 weights are rounded to bf16)
    wide = torch.zeros(19, got.shape[1] + 24, dtype=torch.bfloat16, device="cuda:0")
    ops.linear(x, w, act=act, out=wide[:, 8:8 + got.shape[1]])
    assert rel(wide[:, 8:8 + got.shape[1]], got) < 2.0 ** -8 and float(wide[:, :8].abs().max()) == 0 and float(wide[:, 8 + got.shape[1]:].abs().max()) == 0


@pytest.mark.parametrize("fmt", [WFormat.BF16, WFormat.Q8])
@pytest.mark.parametrize("T,E,k,chunk", [(9, 16, 2, 8), (40, 8, 3, 16), (300, 16, 4, 24), (300, 5, 3, 32), (1000, 3, 2, 40), (33, 300, 8, 16), (64, 4, 1, 64)])
def test_experts_of_a_few_rows(fmt, T, E, k, chunk):
    H, F, dev = 192, 320, "cuda:0"
    gu, down = weight(fmt, F, H, E, 1), weight(fmt, 200, F // 2, E, 2)
    x = torch.randn(T, H, device=dev).to(torch.bfloat16)
    logits = torch.randn(T, E, device=dev) + torch.linspace(0, 3, E, device=dev)
    idx = logits.topk(k, dim=1).indices.int()
    pk = K().moe_pack(idx, E)
    xp = K().moe_gather(x, pk)
    bias = torch.randn(E, F, device=dev)
    a = K().grouped_linear(xp, gu, pk.tile_expert, pk.num_tiles, bias=bias, act=ops.ACT_SWIGLU, out_dtype=torch.float32, tile_valid=pk.tile_valid, chunk=chunk)
    at = pk.pair_to_packed.long()
    e = idx.reshape(-1).long()
    xr = x.double().repeat_interleave(k, 0)
    h = torch.einsum("pk,pnk->pn", xr, values(gu)[e]) + bias.double()[e]
    gate, up = h.view(-1, F // 32, 2, 16).unbind(2)
    want = (torch.nn.functional.silu(gate) * up).reshape(T * k, F // 2)
    assert rel(a[at], want) < 1e-5
    ab = a.to(torch.bfloat16)
    y = K().grouped_linear(ab, down, pk.tile_expert, pk.num_tiles, out_dtype=torch.float32, tile_valid=pk.tile_valid, chunk=chunk)
    assert rel(y[at], torch.einsum("pk,pnk->pn", ab[at].double(), values(down)[e])) < 3e-6


def test_launches_on_two_streams_and_in_a_graph_do_not_share_state():
    x = torch.randn(12, 4096, device="cuda:0").to(torch.bfloat16)
    w = weight(WFormat.BF16, 1024, 4096)
    want = product(x, w, True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = product(x, w, True)
    side = torch.cuda.Stream()
    for _ in range(6):
        graph.replay()
        with torch.cuda.stream(side):
            other = product(x, w, True)
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(other, want)


@pytest.mark.parametrize("M", [3, 5, 8])
@pytest.mark.parametrize("N,Kd", [(6144, 4096), (8192, 2880), (5120, 14336)])
def test_few_rows_in_fp32_lose_nothing_to_the_tensor_cores(M, N, Kd):
    """Sums of 16 products are cut off by 2^-23 of themselves at most and joined with compensation: with independent terms their errors come to no more
    than 2^-23 of the result, rounding included 2^-22.  A running sum kept in the tensor core is cut off K / 16 times: 4e-7 to 3e-6 at these sizes."""
    x = torch.randn(M, Kd, generator=torch.Generator().manual_seed(M)).to("cuda:0", torch.bfloat16)
    w = weight(WFormat.BF16, N, Kd, seed=N)
    assert rel(product(x, w, True), x.double() @ values(w)[0].T) < 2.0 ** -22
    assert rel(ops.linear(x, w, out_f32=True), x.double() @ values(w)[0].T) < 2.0 ** -22


def test_infinite_sums_stay_infinite():
    w = from_dense(torch.rand(1, 6144, 4096, generator=torch.Generator().manual_seed(5)) + 0.5, WFormat.BF16).to("cuda:0")
    x = torch.ones(4, 4096, dtype=torch.bfloat16, device="cuda:0")
    x[0, 7] = float("inf")
    x[1, ::3] = 3e38
    x[2, 4000] = float("nan")
    got = product(x, w, True)
    assert bool(torch.isposinf(got[:2]).all()) and bool(got[2].isnan().all()) and rel(got[3], x[3].double() @ values(w)[0].T) < 2.0 ** -21


@pytest.mark.parametrize("T,E,k,chunk,limit", [(300, 16, 4, 16, 32), (40, 8, 3, 8, 32), (1000, 300, 2, 16, 1), (700, 5, 3, 16, 32), (260, 4, 2, 16, 127), (64, 40, 1, 8, 64)])
def test_experts_of_many_rows_among_experts_of_few(T, E, k, chunk, limit, monkeypatch):
    """Tiles of up to ``limit`` live rows in one kernel, the others in the other one: every pair's row is written once, whatever the order of the two kinds.  The
    bf16 decode of the tcgen05 kernel rounds a weight by 2^-9 of itself: 2^-9 of the sum at most, and less than a third of it with independent terms."""
    monkeypatch.setattr(K(), "expert_rows_max", lambda tokens: limit)
    H, F, dev = 192, 320, "cuda:0"
    gu, down = weight(WFormat.Q8, F, H, E, 1), weight(WFormat.Q8, 200, F // 2, E, 2)
    x = torch.randn(T, H, device=dev).to(torch.bfloat16)
    idx = (torch.randn(T, E, device=dev) + 3 * torch.randn(E, device=dev)).topk(k, dim=1).indices.int()
    pk = K().moe_pack(idx, E)
    xp = K().moe_gather(x, pk)
    bias = torch.randn(E, F, device=dev)
    kw = dict(tile_valid=pk.tile_valid, chunk=chunk, tokens=T, out_dtype=torch.float32)
    a = K().grouped_linear(xp, gu, pk.tile_expert, pk.num_tiles, bias=bias, act=ops.ACT_SWIGLU, **kw)
    at, e = pk.pair_to_packed.long(), idx.reshape(-1).long()
    h = torch.einsum("pk,pnk->pn", x.double().repeat_interleave(k, 0), values(gu)[e]) + bias.double()[e]
    gate, up = h.view(-1, F // 32, 2, 16).unbind(2)
    assert rel(a[at], (torch.nn.functional.silu(gate) * up).reshape(T * k, F // 2)) < 2.0 ** -9
    ab = a.to(torch.bfloat16)
    y = K().grouped_linear(ab, down, pk.tile_expert, pk.num_tiles, **kw)
    assert rel(y[at], torch.einsum("pk,pnk->pn", ab[at].double(), values(down)[e])) < 2.0 ** -9
    assert torch.equal(y[at], K().grouped_linear(ab, down, pk.tile_expert, pk.num_tiles, **kw)[at])
    K().check_status()
