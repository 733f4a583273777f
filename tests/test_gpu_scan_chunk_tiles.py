"""The recurrence in chunks of 128 rows at the bounds of its tiles of 64 rows and of its chunks, and the norm of parts behind it."""

import math

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


@pytest.mark.parametrize("d,silu", [(64, False), (64, True), (128, False), (128, True)])
def test_error_against_64_bits(ops, d, silu):
    """Slow decays, so that all rows of a chunk and the state count.  y passes three sums (scores, q S, P v) of chains of 64
    terms, each off by up to 6.5e-8, all of it towards zero, and their sums over 128 terms and the state's roundings add as much as
    one of them; 128 terms in one chain were off by 5.9e-7 to 6.8e-7 with 128 channels."""
    H, T = 3, 300
    g = torch.Generator().manual_seed(d)
    x = (1.2 * torch.randn(T, 3 * H * d, generator=g)).bfloat16().cuda()
    decay, first = torch.tensor([1 - 2.0 ** -5, 1 - 2.0 ** -8, 1 - 2.0 ** -12], device="cuda"), torch.randn(H, d, d, generator=g).cuda() * 3
    steps = Steps(ops, 1, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
    batch, _ = steps.step({0: T})
    y, state = torch.empty(T, H * d, device="cuda"), steps.mgr.view(0).state["s"]
    slot = int(batch.host.state_slot[0])
    state[slot] = first
    parts = x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:]
    ops.matrix_state_scan(*parts, state, batch, y, H, H, d, d, act_silu=silu, decay=decay, q_scale=0.25)
    ops.check_errors()
    q, k, v = (t.double().view(T, H, d) for t in parts)
    if silu:
        q, k, v = (torch.nn.functional.silu(t) for t in (q, k, v))
    m, want = first.double().transpose(1, 2), torch.empty(T, H, d, dtype=torch.float64, device="cuda")
    for t in range(T):
        m = decay.double()[:, None, None] * m + k[t][:, :, None] * v[t][:, None, :]
        want[t] = torch.einsum("hk,hkv->hv", q[t] * 0.25, m)
    for got, ref in ((y.view(T, H, d), want), (state[slot].transpose(1, 2), m)):
        assert (got.double() - ref).norm() <= 2.6e-7 * ref.norm()


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


def same_kind(got, want):
    """The same infinities and NaN, and finite numbers as near as float32 sums are."""
    fine = want.isfinite()
    assert torch.equal(got.isfinite(), fine) and torch.equal(got[~fine].nan_to_num(0, 1, -1), want[~fine].nan_to_num(0, 1, -1))
    assert (got - want)[fine].norm() <= 1e-6 * want[fine].norm()


@pytest.mark.parametrize("d,silu", [(64, False), (64, True), (128, False), (128, True)])
@pytest.mark.parametrize("what", ["k", "v", "both"])
def test_states_of_infinite_inputs(ops, d, silu, what):
    """Infinities in k and v of rows 3, 70 and 200 leave infinities of the products' signs in the state (NaN where they
    meet zeros or each other), as step by step."""
    H, T = 2, 300
    x = torch.randn(T, 3 * H * d, generator=torch.Generator().manual_seed(2)).bfloat16().cuda()
    for at, value in ((3, float("inf")), (70, float("-inf")), (200, float("inf"))):
        if what != "v":
            x[at, H * d + 5 + at % 7] = value
        if what != "k":
            x[at, 2 * H * d + 9 + at % 5] = value
    (_, got), (_, want) = run(ops, x, [T], H, d, silu), run(ops, x, [T], H, d, silu, prepare=True)
    assert want.isinf().any()
    same_kind(got, want)


@pytest.mark.parametrize("d", [64, 128])
def test_infinities_of_an_earlier_state(ops, d):
    """One infinity and one NaN a head in the state that earlier rows left: every row's y has them with q's sign, as step by step."""
    H, T = 2, 300
    g = torch.Generator().manual_seed(3)
    x, decay = torch.randn(T, 3 * H * d, generator=g).bfloat16().cuda(), torch.tensor([0.99, 0.9], device="cuda")
    out = []
    for prepare in (None, True):
        steps = Steps(ops, 1, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
        batch, _ = steps.step({0: T})
        state, y = steps.mgr.view(0).state["s"], torch.empty(T, H * d, device="cuda")
        slot = int(batch.host.state_slot[0])
        state[slot, :, 7, 11], state[slot, 0, d - 3, 1], state[slot, 1, 2, d - 2] = float("inf"), float("-inf"), float("nan")
        ops.matrix_state_scan(x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:], state, batch, y, H, H, d, d, decay=decay, prepare=prepare)
        out.append((y.double(), state[slot].double()))
    assert (out[1][0] == float("inf")).any() and (out[1][0] == float("-inf")).any()
    for got, want in zip(*out):
        same_kind(got, want)


@pytest.mark.parametrize("d", [64, 128])
def test_a_turned_key_without_parts(ops, d):
    """A key that the rotation leaves between what bfloat16 and what float32 holds, and small values beside it: y and the state are
    finite, as step by step."""
    H, T, at = 2, 300, 150
    g = torch.Generator().manual_seed(4)
    x = torch.randn(T, 3 * H * d, generator=g).bfloat16()
    large = torch.tensor(3.1e38).bfloat16()
    freq = torch.zeros(d // 2, dtype=torch.float64)
    freq[5] = (math.asin(3.4e38 / float(large) / 2 ** 0.5) - math.pi / 4) / at        # (cos + sin) large = 3.4e38
    x[at, H * d + 5], x[at, H * d + 5 + d // 2] = large, large
    x[at, 2 * H * d:] *= 0.01
    x = x.cuda()
    out = []
    for prepare in (None, True):
        steps = Steps(ops, 1, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
        batch, _ = steps.step({0: T})
        state, y = steps.mgr.view(0).state["s"], torch.empty(T, H * d, device="cuda")
        ops.matrix_state_scan(x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:], state, batch, y, H, H, d, d, q_scale=1e-3,
                              decay=torch.tensor([0.99, 0.9], device="cuda"), rotary=(batch.positions, freq.cuda(), d), prepare=prepare)
        out.append((y.double(), state[int(batch.host.state_slot[0])].double()))
    assert all(t.isfinite().all() for pair in out for t in pair) and out[1][1].abs().max() > 1e35
    for got, want in zip(*out):
        same_kind(got, want)
    assert (out[0][0] - out[1][0])[:at].norm() <= 1e-6 * out[1][0][:at].norm()


def test_rows_that_cannot_be_stored_sixteen_bytes_at_a_time(ops):
    """The chunks' kernels store y four floats at a time: a y that stands between goes step by step."""
    H, d, T = 2, 64, 200
    x = torch.randn(T, 3 * H * d, generator=torch.Generator().manual_seed(6)).bfloat16().cuda()
    parts, decay, out = (x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:]), torch.tensor([0.99, 0.9], device="cuda"), []
    for offset, prepare in ((1, None), (0, True)):
        steps = Steps(ops, 1, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
        batch, _ = steps.step({0: T})
        y = torch.zeros(T * H * d + 8, device="cuda")
        state = steps.mgr.view(0).state["s"]
        ops.matrix_state_scan(*parts, state, batch, y[offset:offset + T * H * d].view(T, H * d), H, H, d, d, decay=decay, prepare=prepare)
        assert not y[:offset].any() and not y[offset + T * H * d:].any()
        out.append((y[offset:offset + T * H * d], state))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("T", [1, 3, 41, 400])
@pytest.mark.parametrize("groups,n", [(14, 64), (28, 128), (5, 32), (3, 48), (2, 256)])
def test_norm_of_parts(ops, T, groups, n):
    """Few and many parts, those that go four columns at a time and those that do not, gates in either type and with rows
    further apart: a sum of n squares in float32, then the output type's rounding."""
    C = groups * n
    g = torch.Generator(device="cuda").manual_seed(T + C)
    y = torch.randn(T, C, generator=g, device="cuda")
    for gate_type, out_type, apart, w_len in ((torch.bfloat16, torch.bfloat16, 8, n), (torch.float32, torch.float32, 4, C),
                                              (torch.bfloat16, torch.float32, 2, n), (None, torch.bfloat16, 0, None)):
        gate = None if gate_type is None else torch.randn(T, C + apart, generator=g, device="cuda").to(gate_type)[:, :C]
        w = None if w_len is None else torch.randn(w_len, generator=g, device="cuda")
        out = torch.empty(T, C, dtype=out_type, device="cuda")
        ops.group_rmsnorm_gate(y, gate, w, 1e-5, groups, out, gate_act="silu")
        v = y.double().view(T, groups, n)
        want = (v / (v.square().mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(T, C)
        if w is not None:
            want *= w.double().repeat(C // w_len)
        if gate is not None:
            want *= torch.nn.functional.silu(gate.double())
        tol = 5e-6 if out_type == torch.float32 else 2.0 ** -8
        torch.testing.assert_close(out.double(), want, rtol=tol, atol=1e-6)
