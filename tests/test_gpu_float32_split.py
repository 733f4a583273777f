"""The float32 product in bfloat16 parts (from 512 terms on): the sizes where its kernels and tiles change, in rows, features
and terms; that a row's bits depend on none of them; and operands that have no parts."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


@pytest.mark.parametrize("K", [512, 516, 896, 1024, 1088, 2044, 4864, 20480])
@pytest.mark.parametrize("N", [64, 333, 1152, 5000])
def test_rows_and_error(ops, N, K):
    """Two error bounds for all forms.  An output's: six products of parts leave out at most 2^-24 of a term; a block's last four steps (and
    20 that are 2^-8 as large) lose less than two units of 2^-24 of the terms' magnitudes each, and the sums over
    blocks and ranges round K / 64 + 9 times.  The whole product's, as a share of its norm: a block is off by 6.5e-8 (measured against 64 bits), and
    each of the K / 64 + 9 sums by up to 2^-25 of what it has so far, which add as random signs do; without a
    third part, or without x1 w1, it would be 2.4e-6 or more at every size (computed on the CPU from the parts).  Each row gives the bits that it gives alone."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(700, K, generator=g, device="cuda")
    w, b = torch.randn(N, K, generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda")
    whole = ops.gemm_f32(x, w, b)
    want, size = x.double() @ w.double().T + b.double(), x.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((whole.double() - want).abs() <= (K / 64 + 9 + 8 + 2) * 2.0 ** -24 * size).all()
    assert (whole.double() - want).norm() <= (6.5e-8 + 2.0 ** -25 * (K / 64 + 9) ** 0.5) * want.norm()
    for m in (1, 8, 9, 16, 17, 64, 65, 129, 207, 257, 513):
        assert torch.equal(ops.gemm_f32(x[700 - m:].contiguous(), w, b), whole[700 - m:]), m
    ops.check_errors()


@pytest.mark.parametrize("N,K", [(60, 2048), (16, 2112), (1000, 2112), (2360, 1988), (2384, 2048), (4720, 2052), (4750, 2048), (7120, 2112),
                                 (80, 516), (4720, 1300), (4750, 576), (9480, 516), (9500, 640), (11850, 512), (30000, 900),
                                 (512, 8960), (640, 4868), (900, 3588)])
def test_few_rows_of_every_form(ops, N, K):
    """Forms of the kernels for few rows: with 4 and 8 ranges (the last of them short or empty), tiles that fill the chip once, a
    little more, several times, and clusters.  The bits are those of the kernel for many rows, the batch's those of each."""
    g = torch.Generator(device="cuda").manual_seed(N * K)
    N = max(N, 64)
    x = torch.randn(24, K, generator=g, device="cuda")
    w, b = torch.randn(N, K, generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda")
    whole = ops.gemm_f32(x, w, b)
    assert (whole.double() - (x.double() @ w.double().T + b.double())).norm() <= 2e-7 * whole.double().norm()
    for m in (1, 3, 8, 9, 16):
        assert torch.equal(ops.gemm_f32(x[24 - m:].contiguous(), w, b, constant=True), whole[24 - m:]), m
    if N <= 4800:
        y = ops.head_product(x[:14].view(7, 2, K), torch.stack([w, w.flip(0)]), heads_first=True)
        assert torch.equal(y[1, :5], ops.gemm_f32(x[1:10:2].contiguous(), w.flip(0))) and torch.equal(y[0], ops.gemm_f32(x[:14:2].contiguous(), w))
    ops.check_errors()


@pytest.mark.parametrize("N,K", [(4096, 2048), (4100, 2112), (6144, 3588), (5000, 5000)])
@pytest.mark.parametrize("M", [17, 32, 65, 100])
def test_two_ranges_of_a_cluster(ops, M, N, K):
    """Clusters whose CTAs have two ranges each (the last of them one, where there are seven): the bits of few rows."""
    g = torch.Generator(device="cuda").manual_seed(N + M)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    b = torch.randn(N, generator=g, device="cuda")
    y = ops.gemm_f32(x, w, b)
    for at in range(0, M, 16):
        assert torch.equal(y[at:at + 16], ops.gemm_f32(x[at:at + 16].contiguous(), w, b))
    ops.check_errors()


@pytest.mark.parametrize("M", [3, 11, 40, 300, 1500])
@pytest.mark.parametrize("N", [80, 6000])
def test_operands_without_parts(ops, M, N):
    """Infinities, NaN and numbers that bfloat16 rounds to infinity: the outputs that meet them are what float32
    FMAs give, the others keep their bits."""
    K = 640
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    x[:, 3] *= 0.1                                       # (its product with the largest numbers stays finite)
    before = ops.gemm_f32(x, w)
    x[1, 70], x[2, 71] = float("inf"), 3.4e38
    w[5, 600], w[77, 3] = float("nan"), -3.4e38
    w[5 + 1:, 71].clamp_(-0.5, 0.5)
    w[:, 70].abs_()
    touched = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    touched[1:3], touched[:, 5], touched[:, 77] = True, True, True
    after, clean = ops.gemm_f32(x, w), w.clone()
    clean[5], clean[77] = 0, 0
    rest = ops.gemm_f32(x, clean)
    assert torch.equal(after[~touched], rest[~touched]) and before.isfinite().all()
    assert after[:, 5].isnan().all() and (after[1, 6:77] == float("inf")).all()
    want = (x[2].double() * w[6:77].double()).sum(1)
    torch.testing.assert_close(after[2, 6:77].double(), want, rtol=1e-4, atol=0)
    torch.testing.assert_close(after[0, 77].double(), (x[0].double() * w[77].double()).sum(), rtol=1e-4, atol=0)


def test_products_of_a_batch_and_strided_rows(ops):
    """A product per head over views of wider rows, few rows and many: the bits of each head by itself."""
    H, K, N = 3, 512, 128
    g = torch.Generator(device="cuda").manual_seed(2)
    w = torch.randn(H, N, K, generator=g, device="cuda")
    for T in (5, 200):
        x = torch.randn(T, H * K + 8, generator=g, device="cuda")[:, 4:4 + H * K].view(T, H, K)
        y = ops.head_product(x, w, heads_first=True)
        for h in range(H):
            assert torch.equal(y[h], ops.gemm_f32(x[:, h].contiguous(), w[h]))


def test_rows_that_lie_far_apart(ops):
    """Rows 68 MB apart, of which a tile's last are more than 2^31 floats behind its first."""
    T, K, N, apart = 140, 512, 128, 17_000_000
    x = torch.empty(T * apart, device="cuda").as_strided((T, 1, K), (apart, K, 1))
    g = torch.Generator(device="cuda").manual_seed(3)
    x.copy_(torch.randn(T, 1, K, generator=g, device="cuda"))
    w = torch.randn(1, N, K, generator=g, device="cuda")
    want = x[:, 0].double() @ w[0].double().T
    assert (ops.head_product(x, w, heads_first=True)[0].double() - want).norm() <= 2e-7 * want.norm()


def test_more_rows_than_a_grid_has_tiles(ops):
    """A launch of the kernel for many rows has at most 65,535 tiles of up to 128 rows; the rows behind them are another launch's."""
    M, K, N = 65535 * 128 + 300, 512, 64
    g = torch.Generator(device="cuda").manual_seed(4)
    x, w = torch.zeros(M, K, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    at = torch.cat([torch.arange(40), torch.arange(65535 * 128 - 70, M)]).cuda()
    x[at] = torch.randn(at.numel(), K, generator=g, device="cuda")
    y = ops.gemm_f32(x, w)
    assert torch.equal(y[at], ops.gemm_f32(x[at], w)) and not y[40:65535 * 128 - 70].any()
    ops.check_errors()
