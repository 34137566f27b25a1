"""The gated head norm's vector forms (four rows of up to 128 elements per warp where there are many, two of up to 256) and its general form.  A bf16 result is off by 2^-8 at most."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [4, 30, 64, 96, 128, 132, 256, 260])
@pytest.mark.parametrize("T,n_h,pad", [(1, 1, 0), (3, 5, 4), (7, 2, 1), (2048, 2, 0), (4097, 1, 4), (1639, 3, 0), (1400, 3, 1)])
def test_widths_rows_and_strides(hd, T, n_h, pad):
    from machx_inference_engine_b200.ops import cuda as K
    x = torch.randn(T, n_h * hd, device="cuda:0")
    z = torch.randn(T, n_h * hd + pad, device="cuda:0").to(torch.bfloat16)[:, :n_h * hd]
    w = torch.rand(hd, device="cuda:0") + 0.5
    got = K.gated_rmsnorm_heads(x, z, w, 1e-6, hd).double().view(T, n_h, hd)
    xd, zd = x.double().view(T, n_h, hd), z.double().reshape(T, n_h, hd)
    want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double() * torch.nn.functional.silu(zd)
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8
