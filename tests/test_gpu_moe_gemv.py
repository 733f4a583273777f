"""The matrix-vector product of few entries, where an expert's entries share its rows: counts around the
group of four, entries in any order, identity experts among them, widths that end inside a warp's four
rows, and the widest K (groups of two)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


@pytest.mark.parametrize("tokens,top,E,N,K", [(1, 1, 1, 2, 8), (1, 4, 5, 70, 264), (5, 1, 1, 66, 512), (16, 4, 6, 130, 1000),
                                              (64, 1, 3, 34, 72), (9, 2, 2, 6, 40960), (21, 3, 40, 64, 256)])
@pytest.mark.parametrize("per_token", [True, False])
def test_entries_of_an_expert_share_its_rows(ops, tokens, top, E, N, K, per_token):
    g = torch.Generator().manual_seed(tokens * N)
    n = tokens * top
    table = torch.randint(0, E + (1 if top > 1 else 0), (tokens, top), generator=g, dtype=torch.int32)   # E: identity
    wide = torch.randn(tokens if per_token else n, K, generator=g).bfloat16().cuda()
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    x = wide.repeat_interleave(top, 0) if per_token else wide
    chosen = table.flatten().long()
    live = chosen < E
    want = torch.zeros(n, N, dtype=torch.float64, device="cuda")
    for e in range(n):
        if live[e]:
            want[e] = w[chosen[e]].double() @ x[e].double()
    # float32 sums of K terms: K / 32 in a lane's chain, five more additions
    bound = (K / 32 + 6) * 2.0 ** -24 * max((w[chosen[e]].double().abs() @ x[e].double().abs()).max().item()
                                            for e in range(n) if live[e]) if live.any() else 0.0
    y = ops.moe_gemv(wide, w, None, table.cuda(), per_token=per_token)
    live = live.cuda()
    assert ((y.double() - want).abs()[live] <= bound).all()
    # an entry's bits do not depend on which others there are
    for e in (0, n - 1):
        if live[e]:
            alone = ops.moe_gemv(x[e:e + 1].contiguous(), w, None, table.flatten()[e:e + 1, None].cuda(), per_token=True)
            assert torch.equal(alone[0], y[e])
    form = (7.0, 1.5, 1.0, 0.0)
    act = ops.moe_gemv(wide, w, None, table.cuda(), per_token=per_token, gated=form)
    gate, up = y[:, 0::2].clamp(max=7.0), y[:, 1::2].clamp(-7.0, 7.0)
    glu = gate * torch.sigmoid(1.5 * gate) * (up + 1.0)
    torch.testing.assert_close(act[live].float(), glu[live], rtol=2.0 ** -7, atol=1e-5)
