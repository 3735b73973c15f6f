"""The scratch of the split float32 products: host code, checked without a GPU (where the cut is made for 148 SMs)."""
import pytest

from blackwellllm_b200.kernels import ops


@pytest.mark.parametrize("N,K,shared", [(128, 256, False), (18944, 4096, False), (4096, 4096, True), (57344, 8192, True),
                                        (128256, 4096, True), (152064, 3584, True), (20000, 260, True)])
def test_scratch_is_bounded_whatever_the_weight(N, K, shared):
    per_token, tokens = ops.gemm_f32_scratch(N, K)
    assert (per_token > 0) == shared and 512 <= tokens <= 65535
    assert 4 * per_token * tokens <= 80e6 and 8 * K * tokens <= max(64e6, 8 * K * 512)
    if shared:       # a launch with less, or with none, is refused before anything is queued
        fn = ops._fn("gemm_f32_tc", "bw_gemm_f32_tc", ops._GEMM_F32_TC_ARGS)
        for part, floats in ((16, 5 * per_token - 1), (None, 5 * per_token)):
            assert fn(16, 16, None, 0, 16, 5, N, K, K, N, 0, 16, part, floats, None) == -1
