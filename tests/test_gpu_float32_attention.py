"""The float32 path's attention in bfloat16 parts: the same bits by all its kernels, its error, infinite keys."""

import pytest
import torch

from tests.gpu_util import attention_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


def run(ops, case, nq, nkv, hd, window):
    _, batch, qkv, view, _ = case
    out = torch.full((batch.num_tokens, nq * hd), float("nan"), device="cuda")
    ops.paged_attention(qkv, view.keys, view.values, batch, batch.groups[0], nq, nkv, hd, hd ** -0.5, window, out)
    return out


def copies(ops, n, q, nq, nkv, hd, ps, window, rows, change=None):
    """n requests like each other: cached rows and inputs of all are `rows`."""
    case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=[(131, q)] * n, dtype=torch.float32)
    _, batch, qkv, view, _ = case
    table = batch.groups[0].block_table[:, :-(-(131 + q) // ps)].long()
    for i in range(n):
        live = table[i][table[i] >= 0]
        view.keys[live], view.values[live] = rows[1][:live.numel()], rows[2][:live.numel()]
        if change is not None:
            change(view, table[i])
        qkv[q * i:q * (i + 1)] = rows[0][:q]
    return case


def made(q, nq, nkv, hd, ps):
    g = torch.Generator(device="cuda").manual_seed(hd)
    pages = -(-(131 + q) // ps)
    return (torch.randn(q, (nq + 2 * nkv) * hd, generator=g, device="cuda"),
            torch.randn(pages, nkv, ps, hd, generator=g, device="cuda"), torch.randn(pages, nkv, ps, hd, generator=g, device="cuda"))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("infinite", [False, True])
def test_kernels_give_the_same_bits(ops, hd, window, infinite):
    """Requests of 140 rows: one (18 tiles and heads: four shares), eight (144: two), twenty (360: a warp for 16 rows).  With
    keys that are infinite, so that scores are infinite or NaN, in every kernel what FMAs give."""
    nq, nkv, ps, q = 6, 2, 16, 140
    rows = made(q, nq, nkv, hd, ps)

    def change(view, table):
        if infinite:
            view.keys[table[150 // ps], :, 150 % ps, 3] = float("inf")
            view.keys[table[200 // ps], :, 200 % ps, 5] = -3.4e38
    got = [run(ops, copies(ops, n, q, nq, nkv, hd, ps, window, rows, change), nq, nkv, hd, window) for n in (1, 8, 20)]
    ops.check_errors()
    for out in got:
        for part in out.split(q):
            same = (part == got[0]) | (part.isnan() & got[0].isnan())
            assert same.all()
    if infinite:
        pos, x = torch.arange(131, 131 + q), rows[0][:, :nq * hd].view(q, nq, hd)
        sees = (pos >= 150) & (pos < 150 + (window or 10 ** 6))
        # +infinity takes all (NaN), -infinity takes nothing
        assert got[0].view(q, nq, hd)[sees.cuda()][x[sees.cuda()][:, :, 3] > 0].isnan().all()
        small = sees.cuda() & ~((pos >= 200) & (pos < 200 + (window or 10 ** 6))).cuda()
        assert got[0].view(q, nq, hd)[small][x[small][:, :, 3] < 0].isfinite().all()
        assert got[0][:19].isfinite().all()


@pytest.mark.parametrize("hd,n", [(64, 1), (64, 8), (64, 20), (128, 1), (128, 20)])
def test_error_against_64_bits(ops, hd, n):
    """Scores of a few units are off by a few 2^-24 of the sum of their terms' magnitudes (about 8 times a score), which
    the exponential passes on; the sums over up to 271 keys add less."""
    nq, nkv, ps, q = 6, 2, 16, 140
    rows = made(q, nq, nkv, hd, ps)
    out = run(ops, copies(ops, n, q, nq, nkv, hd, ps, None, rows), nq, nkv, hd, None)[:q].view(q, nq, hd)
    k, v = (t.transpose(1, 2).reshape(-1, nkv, hd)[:131 + q].double() for t in rows[1:])
    s = torch.einsum("qhd,khd->hqk", rows[0][:, :nq * hd].view(q, nq, hd).double(), k.repeat_interleave(nq // nkv, 1)) * hd ** -0.5
    s.masked_fill_(torch.arange(131 + q, device="cuda") > torch.arange(131, 131 + q, device="cuda")[:, None], float("-inf"))
    want = torch.einsum("hqk,khd->qhd", s.softmax(-1), v.repeat_interleave(nq // nkv, 1))
    assert (out.double() - want).norm() <= 1e-6 * want.norm()
    assert (out.double() - want).abs().max() <= 1e-5


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("n", [1, 8])
def test_one_launch_for_portions_and_single_tokens(ops, monkeypatch, hd, window, n):
    """What one launch gives (four shares, two) is what a launch for each gives, bit for bit; more single tokens than the
    rule takes go apart, and so does head size 128."""
    nq, nkv, ps = 6, 2, 16
    for singles in ([0], [63, 64, 700], [500] * 80):
        requests = [(131, 140), (0, 3), *[(0, 64)] * (n - 1)] + [(c, 1) for c in singles]
        if n == 8:
            requests = [(131, 140)] * n + [(c, 1) for c in singles]
        case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=requests, dtype=torch.float32)
        before = ops.launches
        got = run(ops, case, nq, nkv, hd, window)
        took = ops.launches - before
        with monkeypatch.context() as m:
            m.setattr(ops.lib, "somi_attention_f32_mixed_takes", lambda *args: 0)
            want = run(ops, case, nq, nkv, hd, window)
        assert took == (2 if hd == 64 and (len(singles) < 80 or window) else 3)
        assert got.isfinite().all() and torch.equal(got, want)
    ops.check_errors()
