"""The recurrence in chunks of 128 rows at the bounds of its tiles of 64 rows and of its chunks."""

import pytest
import torch

from tests.gpu_util import Steps
from somi_inference_b200.parts.base import StateNeeds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


def run(ops, x, counts, H, d, silu, prepare=None):
    steps = Steps(ops, len(counts), state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
    batch, _ = steps.step(dict(enumerate(counts)))
    y, state = torch.full((batch.num_tokens, H * d), float("nan"), device="cuda"), steps.mgr.view(0).state["s"]
    ops.matrix_state_scan(x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:], state, batch, y, H, H, d, d, act_silu=silu,
                          decay=torch.tensor([0.6, 0.99, 0.9999][:H], device="cuda"), q_scale=0.3, prepare=prepare)
    ops.check_errors()
    return y.double(), state[[int(s) for s in batch.host.state_slot]].double()


@pytest.mark.parametrize("d,silu", [(64, False), (64, True), (128, False), (128, True)])
def test_rows_around_tiles_and_chunks(ops, d, silu):
    """Against the step by step form, which sums the same terms in float32: no further apart than roundings of sums of
    a few hundred terms."""
    H, counts = 3, [193, 255, 256, 257, 319, 320, 321, 384]
    x = torch.randn(sum(counts), 3 * H * d, generator=torch.Generator().manual_seed(d)).bfloat16().cuda()
    for got, want in zip(run(ops, x, counts, H, d, silu), run(ops, x, counts, H, d, silu, prepare=True)):
        assert (got - want).norm() <= 1e-6 * want.norm() and (got - want).abs().max() <= 2e-5 * want.abs().max()


@pytest.mark.parametrize("d,silu", [(64, True), (128, False), (128, True)])
@pytest.mark.parametrize("what", ["v", "k", "q"])
def test_what_is_not_finite_reaches_the_rows_that_see_it(ops, d, silu, what):
    """An infinity and a NaN in row 200 (the second chunk, its second tile): earlier rows keep their bits; of v's column
    the rows from there on are not finite and the other columns keep theirs; of q only that row is touched."""
    H, T, at = 2, 300, 200
    x = torch.randn(T, 3 * H * d, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    y, s = run(ops, x, [T], H, d, silu)
    column = {"q": 0, "k": H * d, "v": 2 * H * d}[what] + 5
    for value in (float("inf"), float("nan")):
        x[at, column] = value
        z, u = run(ops, x, [T], H, d, silu)
        assert torch.equal(z[:at], y[:at]) and torch.equal(z[:, d:], y[:, d:])
        if what == "v":
            assert not z[at:, 5].isfinite().any() and torch.equal(z[:, 6:], y[:, 6:]) and torch.equal(u[0, 0, 6:], s[0, 0, 6:])
        elif what == "k":
            assert not z[at:, :d].isfinite().any() and torch.equal(u[0, :, :, 6:], s[0, :, :, 6:])
        else:
            assert not z[at, :d].isfinite().any() and torch.equal(z[at + 1:], y[at + 1:]) and torch.equal(u, s)
