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
        live = table[i] >= 0                             # (a window's requests have given back the pages behind it)
        view.keys[table[i][live]], view.values[table[i][live]] = rows[1][live], rows[2][live]
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
    if not infinite:
        assert got[0].isfinite().all()                   # (what is not written stays NaN)
    else:
        pos, x = torch.arange(131, 131 + q), rows[0][:, :nq * hd].view(q, nq, hd)
        sees = (pos >= 150) & (pos < 150 + (window or 10 ** 6))
        # +infinity takes all (NaN), -infinity takes nothing
        assert got[0].view(q, nq, hd)[sees.cuda()][x[sees.cuda()][:, :, 3] > 0].isnan().all()
        small = sees.cuda() & ~((pos >= 200) & (pos < 200 + (window or 10 ** 6))).cuda()
        assert got[0].view(q, nq, hd)[small][x[small][:, :, 3] < 0].isfinite().all()
        assert got[0][:19].isfinite().all()


def probabilities(rows, q, nq, nkv, hd, window=None):
    """[nq, q, 131 + q] in 64 bits."""
    k = rows[1].transpose(1, 2).reshape(-1, nkv, hd)[:131 + q].double()
    s = torch.einsum("qhd,khd->hqk", rows[0][:, :nq * hd].view(q, nq, hd).double(), k.repeat_interleave(nq // nkv, 1)) * hd ** -0.5
    key, pos = torch.arange(131 + q, device="cuda"), torch.arange(131, 131 + q, device="cuda")[:, None]
    return s.masked_fill((key > pos) | (key <= pos - (window or 10 ** 6)), float("-inf")).softmax(-1)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38, -3.3962e38])
def test_values_without_parts(ops, hd, window, value):
    """A value that is not finite, or that bfloat16 rounds to infinity, in four shares, two, a warp for 16 rows, and for single
    tokens: rows that do not see it and the other columns keep their bits, those that see it get what FMAs give
    (of a finite one p v, as accurate as p: a few 2^-24 of eight times a score)."""
    nq, nkv, ps, q, at, column = 6, 2, 16, 140, 150, 3
    rows = made(q, nq, nkv, hd, ps)
    clean = run(ops, copies(ops, 1, q, nq, nkv, hd, ps, window, rows), nq, nkv, hd, window).view(q, nq, hd)

    def change(view, table):
        view.values[table[at // ps], :, at % ps, column] = value
    outs = [run(ops, copies(ops, n, q, nq, nkv, hd, ps, window, rows, change), nq, nkv, hd, window) for n in (1, 8, 20)]
    got, pos = outs[0].view(q, nq, hd), torch.arange(131, 131 + q, device="cuda")
    sees = (pos >= at) & (pos < at + (window or 10 ** 6))
    rest = torch.arange(hd, device="cuda") != column
    assert clean.isfinite().all() and torch.equal(got[~sees], clean[~sees]) and torch.equal(got[..., rest], clean[..., rest])
    if abs(value) < float("inf"):
        want = probabilities(rows, q, nq, nkv, hd, window)[:, :, at].T[sees] * value
        torch.testing.assert_close(got[sees][..., column].double(), want, rtol=1e-5, atol=0)
    else:
        assert (got[sees][..., column].isnan() if value != value else got[sees][..., column] == value).all()
    for out in outs[1:]:
        for part in out.view(-1, q, nq, hd):
            assert ((part == got) | (part.isnan() & got.isnan())).all()
    for r in (18, 19, 60, 118, 119, 139):
        case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=[(131 + r, 1)], dtype=torch.float32)
        _, batch, qkv, view, _ = case
        table = batch.groups[0].block_table[0, :-(-(132 + r) // ps)].long()
        live = table >= 0
        view.keys[table[live]], view.values[table[live]] = (t[:table.numel()][live] for t in rows[1:])
        if at // ps < table.numel() and live[at // ps]:
            change(view, table)
        qkv[0] = rows[0][r]
        single = run(ops, case, nq, nkv, hd, window)[0].view(nq, hd)
        assert ((single == got[r]) | (single.isnan() & got[r].isnan())).all()
    ops.check_errors()


@pytest.mark.parametrize("hd,n", [(64, 1), (64, 8), (64, 20), (128, 1), (128, 20)])
def test_error_against_64_bits(ops, hd, n):
    """Scores of a few units are off by a few 2^-24 of the sum of their terms' magnitudes (about 8 times a score), which
    the exponential passes on; the sums over up to 271 keys add less."""
    nq, nkv, ps, q = 6, 2, 16, 140
    rows = made(q, nq, nkv, hd, ps)
    out = run(ops, copies(ops, n, q, nq, nkv, hd, ps, None, rows), nq, nkv, hd, None)[:q].view(q, nq, hd)
    v = rows[2].transpose(1, 2).reshape(-1, nkv, hd)[:131 + q].double()
    want = torch.einsum("hqk,khd->qhd", probabilities(rows, q, nq, nkv, hd), v.repeat_interleave(nq // nkv, 1))
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
