"""The GEMM on pairs of SMs (csrc/cuda/gemm_pair.cu): the values of the one-SM kernel bit for bit (both add the same products in the same order), which is
compared with the oracle elsewhere."""
import ctypes as C

import pytest
import torch

from machx_inference_engine_b200 import _lib, ops
from machx_inference_engine_b200.ops.weights import QuantWeight, WFormat

pytestmark = pytest.mark.gpu


def K():
    from machx_inference_engine_b200.ops import cuda
    return cuda


def pair(x, w, out_kind=0, bias=None, row_scale=None, act=0, pad=0):
    p = K()._p
    n = w.N // 2 if ops.act_gated(act) else w.N
    out = torch.full((x.shape[0], n + pad), 7.0, dtype=(torch.bfloat16, torch.float32, torch.float16)[out_kind], device=x.device)
    rc = _lib.cuda().mx_gemm_pair(p(x), p(w.p0), p(out), out.stride(0), out_kind, p(bias), p(row_scale), act, C.c_float(1.702), C.c_float(7.0), x.shape[0], w.N,
                                  w.K, K()._stream())
    assert rc == 0
    assert pad == 0 or bool((out[:, n:] == 7.0).all())
    return out[:, :n]


@pytest.mark.parametrize("M", [1, 127, 129, 256, 257, 700])
@pytest.mark.parametrize("N,Kd", [(32, 8), (96, 72), (256, 64), (257, 2888), (544, 384), (6144, 512)])
def test_same_values_as_the_one_sm_kernel(M, N, Kd):
    g = torch.Generator(device="cuda:0").manual_seed(M * 7 + N)
    x = torch.randn(M, Kd, generator=g, device="cuda:0").to(torch.bfloat16)
    w = QuantWeight(WFormat.BF16, N, Kd, 1, torch.randn(1, N, Kd, generator=g, device="cuda:0").to(torch.bfloat16))
    bias, rs = torch.randn(N, device="cuda:0"), torch.rand(M, device="cuda:0") + 0.5
    got = pair(x, w, 1)
    want = x.double() @ w.p0[0].double().T
    assert float((got.double() - want).norm() / want.norm()) < 3e-6 + Kd / 16 * 2.0 ** -24      # (fp32 sums, cut off once per 16 products)
    for kw in (dict(), dict(bias=bias), dict(bias=bias, row_scale=rs), dict(act=ops.ACT_RELU2)) + ((dict(act=ops.ACT_SWIGLU, bias=bias),) if N % 32 == 0 else ()):
        for f32 in (0, 1):
            assert torch.equal(pair(x, w, f32, pad=8 if f32 else 3, **kw), K().gemm(x, w, out_f32=bool(f32), bn=128, **kw)), (kw.keys(), f32)


def test_many_tiles_per_cluster_and_two_streams():
    g = torch.Generator(device="cuda:0").manual_seed(3)
    x = torch.randn(2500, 1024, generator=g, device="cuda:0").to(torch.bfloat16)
    w = QuantWeight(WFormat.BF16, 8000, 1024, 1, torch.randn(1, 8000, 1024, generator=g, device="cuda:0").to(torch.bfloat16))
    want = K().gemm(x, w)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(3):
        a = pair(x, w)
        with torch.cuda.stream(side):
            b = pair(x, w)
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b, want)
    assert K()._takes_pair(2500, 8000) and torch.equal(K().linear(x, w), want)
