"""The float32 path's product at the sizes where its kernel changes shape: the bounds of the row tiles
and of the ranges of K; and that a row's bits depend on none of it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


@pytest.mark.parametrize("N", [1, 65, 20000])
@pytest.mark.parametrize("K", [1, 31, 127, 128, 130, 511, 512, 548, 2047, 2048, 2052])
def test_product_at_the_bounds_of_tiles_and_ranges(ops, K, N):
    """Rows around every tile height, K around every change of its ranges, few and many columns (ranges
    over a cluster, ranges one after the other).  A term is rounded at most K / 2 + 9 times, so the error is
    within that many half ulps of the sum of the terms' magnitudes; and each row gives the same bits
    whatever the other rows are."""
    g = torch.Generator().manual_seed(K + N)
    x = torch.randn(130, K, generator=g).cuda()
    w, b = torch.randn(N, K, generator=g).cuda(), torch.randn(N, generator=g).cuda()
    whole = ops.gemm_f32(x, w, b)
    want = x.double() @ w.double().T + b.double()
    bound = (K / 2 + 9) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + b.double().abs())
    assert ((whole.double() - want).abs() <= bound).all()
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65):
        assert torch.equal(ops.gemm_f32(x[130 - m:].contiguous(), w, b), whole[130 - m:]), m
