"""The float32 path's product and attention at the sizes where their kernels change shape: the bounds
of the row tiles, of the ranges of K and of the chunks of keys; and that a row's bits depend on none of it."""

import pytest
import torch

from tests.gpu_util import attention_case, batch_to_cpu
from tests.plain.host_ops import HostOps

pytestmark = pytest.mark.gpu
HOST = HostOps()


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


@pytest.mark.parametrize("N,K", [(65, 548), (9728, 130)])
def test_product_around_the_switch_of_row_tiles(ops, N, K):
    """Up to 384 rows a tile has 32 rows, from there on 64: a row gives the same bits in either."""
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(449, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    whole = ops.gemm_f32(x, w)
    for m in (256, 257, 383, 384, 385):
        assert torch.equal(ops.gemm_f32(x[:m].contiguous(), w), whole[:m]), m


def test_product_with_more_rows_than_a_grid_has_tiles(ops):
    """65,535 tiles of 64 rows and 70 rows more: each product is a sum of four terms (five roundings)."""
    g = torch.Generator(device="cuda").manual_seed(3)
    M, K, N = 65535 * 64 + 70, 4, 3
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    y, bound = ops.gemm_f32(x, w), 5 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((y.double() - x.double() @ w.double().T).abs() <= bound).all()


def run(ops, case, nq, nkv, hd, window):
    mgr, batch, qkv, view, order = case
    out = torch.full((batch.num_tokens, nq * hd), float("nan"), device="cuda")
    ops.paged_attention(qkv, view.keys, view.values, batch, batch.groups[0], nq, nkv, hd, hd ** -0.5, window, out)
    return out


@pytest.mark.parametrize("nq,nkv,hd,ps,window", [(14, 2, 64, 16, None), (3, 3, 128, 8, None), (18, 2, 64, 32, 70),
                                                 (16, 1, 128, 16, 64), (4, 2, 64, 16, 1)])
def test_attention_at_the_bounds_of_chunks(ops, nq, nkv, hd, ps, window):
    """Portions and single tokens that end on, before and behind a chunk of 64 keys and a tile of 64 rows."""
    reqs = [(0, 2), (0, 63), (0, 64), (1, 64), (0, 65), (63, 2), (130, 129), (0, 1), (62, 1), (63, 1), (64, 1),
            (65, 1), (127, 1), (128, 1), (700, 1)]
    case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=reqs, dtype=torch.float32)
    mgr, batch, qkv, view, _ = case
    out = run(ops, case, nq, nkv, hd, window)
    ref = torch.empty_like(out, device="cpu")
    host = batch_to_cpu(batch)
    HOST.paged_attention(qkv.cpu(), view.keys.cpu(), view.values.cpu(), host, host.groups[0], nq, nkv, hd,
                         hd ** -0.5, window, ref)
    # both sides are float32: a few hundred roundings of values about 1
    torch.testing.assert_close(out.cpu(), ref, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("window", [None, 100])
def test_attention_does_not_depend_on_the_cut(ops, window):
    """The last 140 rows of a request of 271 give the same bits as one portion, and each as a single token."""
    nq, nkv, hd = 6, 2, 64
    whole = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=16, window=window, requests=[(131, 140)],
                           dtype=torch.float32, seed=1)
    store, table = whole[3], whole[1].groups[0].block_table[0]
    want = run(ops, whole, nq, nkv, hd, window)
    for r in (0, 60, 61, 139):
        mgr, batch, qkv, view, _ = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=16, window=window,
                                                  requests=[(131 + r, 1)], dtype=torch.float32, seed=2)
        n = -(-(132 + r) // 16)
        live = batch.groups[0].block_table[0, :n] >= 0
        for mine, theirs in ((view.keys, store.keys), (view.values, store.values)):
            mine[batch.groups[0].block_table[0, :n][live].long()] = theirs[table[:n][live].long()]
        qkv.copy_(whole[2][r:r + 1])
        got = run(ops, (mgr, batch, qkv, view, None), nq, nkv, hd, window)
        assert torch.equal(got[0], want[r]), r


@pytest.mark.parametrize("window", [None, 40])
def test_a_later_value_that_is_infinite_reaches_no_earlier_row(ops, window):
    """The value of position 150 is infinite: rows in front of it (in its chunk and tile, too) and, under the
    window, rows that have passed it keep their bits."""
    nq, nkv, hd = 4, 2, 64
    case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=16, window=window, requests=[(100, 120)], dtype=torch.float32)
    want = run(ops, case, nq, nkv, hd, window)
    table = case[1].groups[0].block_table[0]
    case[3].values[int(table[150 // 16]), :, 150 % 16] = float("inf")
    got = run(ops, case, nq, nkv, hd, window)
    sees = torch.arange(100, 220) >= 150
    if window:
        sees &= torch.arange(100, 220) < 150 + window
    assert torch.equal(got[~sees.cuda()], want[~sees.cuda()])
    assert not got[sees.cuda()].isfinite().any()


def test_product_with_a_matrix_made_in_the_same_step(ops):
    """`w` is an output of the kernel in front: without `constant` it is read behind that kernel."""
    g = torch.Generator().manual_seed(4)
    a, b, x = (torch.randn(n, 256, generator=g).cuda() for n in (256, 300, 5))
    for _ in range(20):
        w = ops.gemm_f32(b, a, constant=True)
        y = ops.gemm_f32(x, w)
        torch.testing.assert_close(y.double(), x.double() @ w.double().T, rtol=1e-4, atol=1e-2)


@pytest.mark.parametrize("hd", [64, 128, 32])
@pytest.mark.parametrize("window", [None, 67])
@pytest.mark.parametrize("at", [0, 63, 64, 128])
def test_a_score_that_is_no_number_reaches_every_row_that_sees_it(ops, hd, window, at):
    """The key of position `at` is NaN: also where it is the only visible key of its chunk (the row at a chunk's
    first position, a window's last key), the rows that see it are NaN, and the others keep their bits.  (Head size
    32 runs the kernel for any size.)"""
    nq, nkv, ps = 4, 2, 16
    reqs = [(0, 200), (60, 10)] + [(n, 1) for n in (0, 63, 64, 128, 129, 130, 150)]
    case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=reqs, dtype=torch.float32)
    batch = case[1]
    want = run(ops, case, nq, nkv, hd, window)
    sees, tables = [], batch.groups[0].block_table.cpu()
    for i, (c, q) in enumerate(reqs):
        page = int(tables[i, at // ps]) if at < c + q else -1
        if page >= 0:                                    # (a window has taken back what nobody sees)
            case[3].keys[page, :, at % ps] = float("nan")
        sees += [at <= p and (window is None or at > p - window) for p in range(c, c + q)]
    sees = torch.tensor(sees).cuda()
    got = run(ops, case, nq, nkv, hd, window)
    assert got[sees].isnan().all()
    assert torch.equal(got[~sees], want[~sees])


@pytest.mark.parametrize("window", [None, 1, 65, 70])
def test_attention_of_single_tokens_in_groups(ops, monkeypatch, window):
    """Requests one group behind the other over the same scratch: the same bits as all in one launch."""
    nq, nkv, hd = 6, 2, 64
    reqs = [(0, 70)] + [(n, 1) for n in (0, 63, 64, 65, 127, 128, 129, 130, 700)]
    case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=16, window=window, requests=reqs, dtype=torch.float32)
    want = run(ops, case, nq, nkv, hd, window)
    for requests in (1, 2, 4):
        monkeypatch.setattr(ops, "F32_PART_FLOATS", requests * nq * (12 if window is None else (window + 62) // 64 + 1) * (hd + 2))
        assert torch.equal(run(ops, case, nq, nkv, hd, window), want)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window,infinite", [(None, False), (100, False), (None, True), (100, True)])
def test_shares_of_a_tile_give_the_same_bits(ops, hd, window, infinite):
    """A tile of 64 rows is one CTA's, or shared by two or four where a step has few: a request of 140 rows alone
    (18 tiles and heads: four), among 5 (90: two) and among 20 like it (360: one), with an infinite value too."""
    nq, nkv, ps = 6, 2, 16
    got, first = [], None
    for n in (1, 5, 20):
        case = attention_case(ops, nq=nq, nkv=nkv, hd=hd, page_size=ps, window=window, requests=[(131, 140)] * n,
                              dtype=torch.float32)
        _, batch, qkv, view, _ = case
        assert batch.tiles[64].shape[0] * nq == 18 * n
        table = batch.groups[0].block_table[:, :17].long()
        if first is None:
            if infinite:
                view.values[table[0, 150 // ps], :, 150 % ps] = float("inf")
            live = table[0] >= 0
            first = qkv.clone(), view.keys[table[0][live]].clone(), view.values[table[0][live]].clone()
        for i in range(n):
            assert torch.equal(table[i] >= 0, live)
            view.keys[table[i][live]], view.values[table[i][live]] = first[1], first[2]
            qkv[140 * i:140 * (i + 1)] = first[0]
        got.append(run(ops, case, nq, nkv, hd, window))
    sees = torch.arange(131, 271) >= 150
    if window:
        sees &= torch.arange(131, 271) < 150 + window
    for out in got:
        for part in out.split(140):
            assert torch.equal(part[~sees.cuda()], got[0][~sees.cuda()])
            if not infinite:
                assert torch.equal(part, got[0])
            else:
                assert not part[sees.cuda()].isfinite().any()
