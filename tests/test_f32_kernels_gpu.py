"""The 32-bit path's products for a few tokens, at the edges of their tiles, against 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from blackwellllm_b200.kernels import ops as o
    return o


def rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def product_error(out, x, w, *more):
    ref = x.double() @ w.double().T
    size = math.sqrt(x.shape[1]) * float(x.double().pow(2).mean().sqrt() * w.double().pow(2).mean().sqrt())
    for m in more:
        ref = ref + m.double()
    return float((out.double() - ref).abs().max()) / size


# tokens on both sides of each of the kernel's sizes; features that leave the last block ragged; channels from one lane's four to
# several steps of all warps and a part of one
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(1, 4), (7, 132), (130, 1024), (64, 1028), (9, 4100)])
def test_few_tokens(ops, M, N, K):
    x, w, b, base = rand(M, K, seed=1), rand(N, K, seed=2), rand(N, seed=3), rand(M, N, seed=4)
    out = ops.gemm_simt(x, w, b, out=base.clone(), accumulate=True)
    # a lane adds K / 1024 * 4 products in a row, then 13 partial sums: the error of that many float32 roundings
    bound = 2 ** -24 * (K / 256 + 16) * 4
    assert product_error(out, x, w, b, base) <= bound
    assert product_error(ops.gemm_simt(x, w, b.bfloat16()), x, w, b.bfloat16()) <= bound
    one = ops.gemm_simt(x[M - 1:], w)
    assert torch.equal(ops.gemm_simt(x, w)[M - 1:], one)       # a token's sum is the same whatever is beside it
    wide = rand(M, K + 12, seed=5)
    assert product_error(ops.gemm_simt(wide[:, 4:4 + K], w), wide[:, 4:4 + K], w) <= bound      # rows further apart
    # rows that do not begin on 16 bytes: the general kernel
    assert product_error(ops.gemm_simt(wide[:, 3:3 + K], w), wide[:, 3:3 + K], w) <= 2 ** -24 * K
