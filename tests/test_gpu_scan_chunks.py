"""The recurrence with a constant decay in chunks of 128 rows, against the recurrence itself in 64 bits and
against the step by step kernel: portions that end around a chunk, states that an earlier step left, single
tokens beside them, rotated or activated inputs, grouped query and key heads."""

import pytest
import torch

from tests.gpu_util import Steps
from somi_inference_b200.parts.base import StateNeeds

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


def turned(x, pos, freq):
    half = freq.numel()
    angle = pos.double()[:, None, None] * freq
    c, s, a, b = torch.cos(angle), torch.sin(angle), x[..., :half], x[..., half:2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], -1)


@pytest.mark.parametrize("H,G,d,rot,silu", [(3, 3, 128, 128, False), (4, 2, 64, 0, True), (2, 2, 64, 16, False), (2, 1, 128, 0, False)])
def test_portions_in_chunks(ops, H, G, d, rot, silu):
    g = torch.Generator().manual_seed(d + rot)
    steps = Steps(ops, 6, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16, max_len=2048)
    decay = torch.tensor([0.5, 0.97, 0.9995, 1.0][:H])
    freq = 10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64) / max(1, rot // 2))
    states = torch.zeros(6, H, d, d, dtype=torch.float64)
    state = steps.mgr.view(0).state["s"]
    for counts in ({0: 63, 1: 64, 2: 65, 3: 200, 4: 2, 5: 1000}, {0: 1, 1: 128, 2: 67, 3: 257, 4: 1, 5: 64}):
        batch, where = steps.step(counts)
        T = batch.num_tokens
        x = torch.randn(T, 2 * G * d + H * d, generator=g).bfloat16()
        q, k, v = x[:, :G * d].cuda(), x[:, G * d:2 * G * d].cuda(), x[:, 2 * G * d:].cuda()
        args = (q, k, v)
        kw = dict(act_silu=silu, q_scale=0.25, decay=decay.cuda(),
                  rotary=(batch.positions, freq.cuda(), rot) if rot else None)
        assert ops.scan_in_chunks(*args, batch, H, G, d, d, silu, None, None, None, kw["rotary"])
        y, before = torch.full((T, H * d), float("nan"), device="cuda"), state.clone()
        ops.matrix_state_scan(*args, state, batch, y, H, G, d, d, **kw)
        by_step, s_step = torch.empty_like(y), before.clone()
        ops.matrix_state_scan(*args, s_step, batch, by_step, H, G, d, d, prepare=True, **kw)
        want = torch.empty(T, H, d, dtype=torch.float64)
        act = torch.nn.functional.silu if silu else (lambda t: t)
        for r, (row, n, ctx) in where.items():
            xs = x[row:row + n].double()
            qq, kk, vv = (t.reshape(n, -1, d) for t in (xs[:, :G * d], xs[:, G * d:2 * G * d], xs[:, 2 * G * d:]))
            pos = torch.arange(ctx, ctx + n)
            qq, kk, vv = act(turned(qq, pos, freq)) * 0.25, act(turned(kk, pos, freq)), act(vv)
            qq, kk = qq.repeat_interleave(H // G, 1), kk.repeat_interleave(H // G, 1)
            m = states[r]
            for t in range(n):
                m = decay.double()[:, None, None] * m + kk[t][:, :, None] * vv[t][:, None, :]
                want[row + t] = torch.einsum("hk,hkv->hv", qq[t], m)
            states[r] = m
        slots = {r: int(batch.host.state_slot[j]) for j, r in enumerate(batch.host.requests)}
        want = want.reshape(T, -1)
        got_s = torch.stack([state[slots[r]].double().cpu().transpose(1, 2) for r in range(6)])
        step_s = torch.stack([s_step[slots[r]].double().cpu().transpose(1, 2) for r in range(6)])
        # float32 sums either way: no further off than the step by step form by more than a few roundings
        for got, step, ref in ((y.double().cpu(), by_step.double().cpu(), want), (got_s, step_s, states)):
            off, limit = (got - ref).norm() / ref.norm(), (step - ref).norm() / ref.norm()
            assert off <= 1.5 * limit + 2e-7, (off, limit)
            assert (got - ref).abs().max() <= 2e-5 * ref.abs().max()


def test_a_later_value_that_is_infinite_reaches_no_earlier_row(ops):
    H, d, T = 2, 64, 200
    g = torch.Generator().manual_seed(9)
    x, decay = torch.randn(T, 3 * H * d, generator=g).bfloat16().cuda(), torch.full((H,), 0.9, device="cuda")
    out = []
    for value in (None, float("inf")):
        steps = Steps(ops, 1, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
        batch, _ = steps.step({0: T})
        if value is not None:
            x[75, 2 * H * d:] = value
        y = torch.empty(T, H * d, device="cuda")
        q, k, v = x[:, :H * d], x[:, H * d:2 * H * d], x[:, 2 * H * d:]
        assert ops.scan_in_chunks(q, k, v, batch, H, H, d, d, False, None, None, None, None)
        ops.matrix_state_scan(q, k, v, steps.mgr.view(0).state["s"], batch, y, H, H, d, d, decay=decay)
        out.append(y)
    assert torch.equal(out[0][:75], out[1][:75]) and not out[1][75].isfinite().any()


@pytest.mark.parametrize("d,rot", [(64, 64), (128, 0)])
def test_a_portion_alone_gives_the_same_bits(ops, d, rot):
    """Portions that go in chunks between such as do not, and single tokens: outputs and states are those of the
    request by itself."""
    H, counts = 2, {0: 2, 1: 300, 2: 63, 3: 128, 4: 30, 5: 257, 6: 1}
    g = torch.Generator().manual_seed(d)
    decay, freq = torch.tensor([0.9, 0.999]).cuda(), (10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64) / 64)).cuda()
    x = {r: torch.randn(n, 3 * H * d, generator=g).bfloat16().cuda() for r, n in counts.items()}

    def run(which):
        steps = Steps(ops, 7, state=StateNeeds({"s": ((H, d, d), torch.float32)}), dtype=torch.bfloat16)
        batch, where = steps.step({r: counts[r] for r in which})
        rows = torch.cat([x[r] for r in which if counts[r] > 1] + [x[r] for r in which if counts[r] == 1])
        y, state = torch.full((rows.shape[0], H * d), float("nan"), device="cuda"), steps.mgr.view(0).state["s"]
        ops.matrix_state_scan(rows[:, :H * d], rows[:, H * d:2 * H * d], rows[:, 2 * H * d:], state, batch, y, H, H, d, d,
                              decay=decay, rotary=(batch.positions, freq, rot) if rot else None)
        slots = dict(zip(batch.host.requests, batch.host.state_slot))
        return {r: (y[where[r][0]:where[r][0] + counts[r]], state[int(slots[r])]) for r in which}
    together = run(list(counts))
    for r in counts:
        for a, b in zip(together[r], run([r])[r]):
            assert torch.equal(a, b), r
