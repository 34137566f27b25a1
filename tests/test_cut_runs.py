"""Host arithmetic of the kernels that cut a list of work into equal runs (csrc/cuda/gemm_rows.cu, attention_decode.cu): run lengths and the sizes that their
32-bit counts hold.  The kernels call the same functions."""
import math

import pytest

from machx_inference_engine_b200 import _build, _lib


@pytest.fixture(scope="module")
def lib():
    if not _build.CUDA_LIB.exists() and _build._nvcc() is None:
        pytest.skip("no kernel library and no compiler")
    return _lib.cuda()


@pytest.mark.parametrize("total", [1, 7, 295, 296, 297, 3_500_000, 3_600_000, 4_128_768, 40_000_000, 2 ** 30 - 1])
@pytest.mark.parametrize("steps_nt,cost", [(1, 1), (64, 6), (112, 9), (2688, 21)])
def test_a_product_is_cut_into_equal_runs_of_any_length(lib, total, steps_nt, cost):
    want = max(-(-total // 296), cost, math.isqrt(-(-steps_nt // 15) - 1) + 1 if steps_nt > 15 else 1)
    assert lib.mx_gemm_rows_run(total, 296, steps_nt, cost) == want      # (256 experts of 4096 x 7168 with 16 rows each are 4.1 M units: 13949 per CTA)


@pytest.mark.parametrize("total,most", [(0, 0), (1, 1), (100, 3), (296, 64), (512 * 2048 * 8, 2048), (5_000_000, 2048), (2 ** 31 - 1, 16384)])
def test_attention_tiles_are_cut_into_equal_runs_of_any_length(lib, total, most):
    want = max(-(-total // 296), 1, math.isqrt(max(-(-most // 8) - 1, 0)) + (most > 8))
    assert lib.mx_attention_decode_run(total, 296, most) == want


def test_banks_past_the_counts_are_left_to_the_other_kernel(lib):
    bf16, q8 = 0, 1
    takes = lib.mx_gemm_rows_takes
    assert takes(q8, 586, 16, 1024, 2048) and takes(q8, 256, 16, 4096, 7168) and takes(bf16, 1024, 64, 4096, 4096)
    assert not takes(q8, 1025, 16, 128, 128) and not takes(q8, 10, 65, 128, 128) and not takes(q8, 10, 0, 128, 128)
    assert not takes(q8, 1024, 8, 28672, 8192)                           # 16 groups of 7 units, 224 x 64 steps
    for chunk in (1, 8, 16, 24, 64):
        for tiles in (1, 8, 334, 1024):
            for N, K in ((128, 128), (4096, 7168), (28672, 4096), (151936, 8192)):
                units = tiles * -(-128 // chunk) * (5 + 2 * -(-chunk // 8)) * -(-N // 128) * -(-K // 128)
                assert bool(takes(q8, tiles, chunk, N, K)) == (units < 2 ** 30)
