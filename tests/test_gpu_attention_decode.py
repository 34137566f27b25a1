"""Decode attention on the tensor cores (csrc/cuda/attention_decode.cu) against the fp32 oracle and the general CUDA-core kernel.

Bound of the comparisons: both sides see the same bf16 / int8 operands and sum in fp32; the result is rounded to bf16 once (relative 2^-8 =
3.9e-3 at most), the oracle keeps fp32."""
import pytest
import torch

from machx_inference_engine_b200.ops import ref

pytestmark = pytest.mark.gpu
TOL = 4e-3


def K():
    from machx_inference_engine_b200.ops import cuda
    return cuda


def case(q_lens, kv_lens, n_q, n_kv, hd, bs=128, seed=0, q_pad=0):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    nb = max((n + bs - 1) // bs for n in kv_lens)
    B = len(kv_lens)
    kc, vc = (torch.randn(B * nb + 1, n_kv, bs, hd, generator=g, device=dev).to(torch.bfloat16) for _ in "kv")
    bt = (torch.randperm(B * nb, generator=g, device=dev) + 1).int().view(B, nb)
    cu = torch.tensor([0] + q_lens, device=dev).cumsum(0).int()
    wide = torch.randn(sum(q_lens), n_q * hd + q_pad, generator=g, device=dev).to(torch.bfloat16)
    return wide[:, :n_q * hd].unflatten(1, (n_q, hd)), kc, vc, bt, torch.tensor(kv_lens, dtype=torch.int32, device=dev), cu


def int8_rows(c):
    f = c.float()
    sc = f.abs().amax(-1).clamp_min(1e-6) / 127.0
    return torch.round(f / sc.unsqueeze(-1)).clamp(-128, 127).to(torch.int8), sc


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


SHAPES = [(64, 64, 8), (64, 16, 1), (64, 7, 7), (128, 32, 8), (128, 24, 8), (128, 32, 1), (256, 16, 2), (256, 32, 2), (256, 6, 2)]


@pytest.mark.parametrize("hd,n_q,n_kv", SHAPES)
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("window,keep", [(0, 0), (128, 0), (100, 70)])
def test_decode_lengths_around_the_tiles(hd, n_q, n_kv, int8, window, keep):
    if int8 and keep:
        keep = 0                                                # the int8 cache has no kept keys
    lens = [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 700, 2049]
    q, kc, vc, bt, sl, cu = case([1] * len(lens), lens, n_q, n_kv, hd)
    sinks = torch.randn(n_q, device=q.device)
    scales = None
    if int8:
        (kc, ks), (vc, vs) = int8_rows(kc), int8_rows(vc)
        scales = (ks, vs)
    want = ref.attention(q, kc, vc, bt, sl, cu, 1, sinks=sinks, window=window, keep_first=keep, kv_scales=scales)
    got = K().attention(q.contiguous(), kc, vc, bt, sl, cu, 1, sinks=sinks, window=window, keep_first=keep, kv_scales=scales)
    assert rel(got, want) < TOL
    general = K().attention(q.contiguous(), kc, vc, bt, sl, cu, 1, sinks=sinks, window=window, keep_first=keep, kv_scales=scales, n_splits=3)
    assert rel(got, general) < 2 * TOL
    again = K().attention(q.contiguous(), kc, vc, bt, sl, cu, 1, sinks=sinks, window=window, keep_first=keep, kv_scales=scales)
    assert torch.equal(got, again)


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 64, 8), (128, 32, 8), (256, 16, 2), (128, 5, 5)])
@pytest.mark.parametrize("bs", [64, 128])
def test_short_query_segments(hd, n_q, n_kv, bs):
    q_lens, kv_lens = [2, 1, 0, 63, 9, 40], [2, 300, 128, 63, 1000, 515]
    q, kc, vc, bt, sl, cu = case(q_lens, kv_lens, n_q, n_kv, hd, bs=bs, q_pad=24, seed=3)
    Tq = q.shape[0]
    sinks, gate = torch.randn(n_q, device=q.device), torch.randn(Tq, n_q * hd, device=q.device).to(torch.bfloat16)
    factor = torch.rand(600, device=q.device) + 0.5
    factor_all = torch.cat([factor, factor[-1:].expand(600)])
    for kw in (dict(), dict(sinks=sinks, softcap=20.0), dict(gate=gate, window=70), dict(gate=gate[:, :n_q], sinks=sinks), dict(q_scale=factor)):
        rkw = dict(kw, q_scale=factor_all) if "q_scale" in kw else kw
        got = K().attention(q, kc, vc, bt, sl, cu, 63, **kw)
        assert rel(got, ref.attention(q, kc, vc, bt, sl, cu, 63, **rkw)) < TOL, list(kw)


def test_groups_cut_over_many_parts_and_one_long_sequence_among_short_ones():
    for hd, n_q, n_kv, lens in ((256, 8, 1, [40000]), (64, 8, 1, [30011]), (128, 32, 8, [9000] + [3] * 100), (64, 64, 8, list(range(1, 500, 8)))):
        q, kc, vc, bt, sl, cu = case([1] * len(lens), lens, n_q, n_kv, hd, seed=5)
        assert rel(K().attention(q, kc, vc, bt, sl, cu, 1), ref.attention(q, kc, vc, bt, sl, cu, 1)) < TOL, (hd, len(lens))


def test_rows_past_the_end_are_not_read_and_large_scores_stay_finite():
    q, kc, vc, bt, sl, cu = case([1, 1], [70, 133], 8, 2, 128, seed=7)
    want = K().attention(q, kc, vc, bt, sl, cu, 1)
    for b, n in enumerate(sl.tolist()):                         # what lies behind a sequence's last key does not matter, whatever it holds
        page = int(bt[b, (n - 1) // 128])
        kc[page, :, (n - 1) % 128 + 1:] = float("nan")
        vc[page, :, (n - 1) % 128 + 1:] = float("inf")
    assert torch.equal(K().attention(q, kc, vc, bt, sl, cu, 1), want)
    q, kc, vc, bt, sl, cu = case([1, 1], [700, 133], 8, 2, 64, seed=8)
    kc.mul_(300.0)
    got = K().attention(q, kc, vc, bt, sl, cu, 1)
    assert torch.isfinite(got.float()).all() and rel(got, ref.attention(q, kc, vc, bt, sl, cu, 1)) < 2e-2   # (scores near 1e3: fp32 exponents off by 1e-4)


def test_more_groups_than_the_list_holds_take_the_general_kernel():
    q, kc, vc, bt, sl, cu = case([1] * 520, [5] * 520, 8, 2, 64, bs=64, seed=9)
    assert rel(K().attention(q, kc, vc, bt, sl, cu, 1), ref.attention(q, kc, vc, bt, sl, cu, 1)) < TOL


def test_graph_replays_while_another_stream_decodes():
    q, kc, vc, bt, sl, cu = case([1] * 3, [900, 37, 4000], 32, 8, 128, seed=11)
    want = K().attention(q, kc, vc, bt, sl, cu, 1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = K().attention(q, kc, vc, bt, sl, cu, 1)
    side = torch.cuda.Stream()
    for _ in range(4):
        graph.replay()
        with torch.cuda.stream(side):
            other = K().attention(q, kc, vc, bt, sl, cu, 1)
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(other, want)
