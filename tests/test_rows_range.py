"""Which dense layers of a few rows take the weight-streaming kernel: sizes at which another kernel was measured to be faster stay with it."""
import pytest
import torch

from machx_inference_engine_b200 import _build
from machx_inference_engine_b200.ops import cuda as K
from machx_inference_engine_b200.ops.weights import QuantWeight, WFormat

B, Q = WFormat.BF16, WFormat.Q8
# format, rows, columns, depth, gated
OTHER_KERNEL = [(B, 3, 256, 4096, 0), (B, 8, 64, 2048, 0), (B, 4, 3072, 2048, 0), (B, 6, 1024, 4096, 0), (B, 48, 1000, 264, 0), (B, 32, 2048, 2048, 0), (B, 48, 12288, 2048, 0),
                (B, 33, 2880, 4096, 0), (B, 32, 4096, 2048, 0), (B, 28, 4096, 1024, 0), (B, 48, 6144, 1024, 0), (B, 2, 6144, 4096, 0), (B, 33, 32768, 4096, 0), (B, 32, 2048, 2048, 1),
                (B, 48, 4096, 2048, 1), (B, 48, 192, 512, 1), (Q, 3, 4096, 2048, 0), (Q, 40, 2048, 512, 0), (Q, 41, 6144, 4096, 0), (Q, 2, 8192, 4096, 1), (Q, 3, 4096, 2048, 1), (Q, 4, 2048, 2048, 1)]
THIS_KERNEL = [(B, 40, 6144, 4096, 0), (B, 3, 6144, 4096, 0), (B, 3, 8192, 512, 0), (B, 8, 4096, 4096, 0), (B, 9, 64, 2048, 0), (B, 24, 2048, 2048, 0), (B, 32, 28672, 4096, 1), (B, 2, 28672, 4096, 1),
               (B, 48, 4096, 14336, 0), (B, 48, 128, 2880, 0), (B, 31, 3072, 2048, 0), (B, 40, 2048, 2048, 1), (Q, 40, 6144, 4096, 0), (Q, 4, 4096, 2048, 0), (Q, 3, 1024, 4096, 0),
               (Q, 2, 28672, 4096, 1), (Q, 8, 1024, 2048, 1)]


@pytest.fixture(autouse=True)
def b200(monkeypatch):
    monkeypatch.setattr(K, "_sm_count", 148)


@pytest.mark.parametrize("case,here", [(c, False) for c in OTHER_KERNEL] + [(c, True) for c in THIS_KERNEL])
def test_measured_sizes(case, here):
    fmt, M, N, Kd, gated = case
    fewest, most = K._rows_range(fmt, M, N, Kd, bool(gated))
    assert (fewest <= M <= most) == here


def test_pairs_of_sms_stay_away_from_short_sums_in_few_tiles():
    for M, N, Kd, here in ((640, 2048, 512, False), (200, 8192, 1536, False), (640, 2048, 2048, True), (1024, 4096, 256, True), (4096, 28672, 4096, True), (256, 4096, 4096, False)):
        assert K._takes_pair(M, N, Kd) == here, (M, N, Kd)


@pytest.mark.skipif(not _build.CUDA_LIB.exists() and _build._nvcc() is None, reason="no kernel library and no compiler")
def test_a_gemv_path_that_is_asked_for_is_the_one_that_runs():
    x, w = torch.zeros(8, 4096, dtype=torch.bfloat16), QuantWeight(B, 4096, 4096, 1, torch.zeros(1, 4096, 4096, dtype=torch.bfloat16))
    assert K._takes_rows(x, w, 0, None)
    try:
        for path in ("stream", "register"):
            K.set_gemv_path(path)
            assert not K._takes_rows(x, w, 0, None), path
    finally:
        K.set_gemv_path("auto")
    assert K._takes_rows(x, w, 0, None)


@pytest.mark.parametrize("M", [3, 5, 6, 7])
def test_long_rows_leave_the_gemv_only_while_it_serves_them_badly(M, monkeypatch):
    x, w = torch.zeros(M, 12288, dtype=torch.bfloat16), QuantWeight(B, 64, 12288, 1, torch.zeros(1, 64, 12288, dtype=torch.bfloat16))
    assert K._takes_rows(x, w, 0, None) == K._few_rows_take_gemm(M, w, 0) == (M > 5)
    monkeypatch.setattr(K, "_few_rows_take_gemm", lambda *a: False)
    assert not K._takes_rows(x, w, 0, None)
