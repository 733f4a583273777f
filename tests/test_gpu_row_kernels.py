"""The kernels around a layer's products where they change shape: the norm of many rows at the ends of its
vectors, the rotary kernels around their tokens per CTA, the merge of decode attention around its loads."""

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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [4, 508, 516, 3584, 8192, 8196, 37])
def test_norm_of_many_rows(ops, dtype, H):
    """33 rows and more; 8,192 columns are the widest of the kernel of many rows, 8,196 and 37 run another."""
    g = torch.Generator().manual_seed(H)
    res, delta = torch.randn(40, H, generator=g), torch.randn(40, H, generator=g).to(dtype)
    w = (1 + 0.3 * torch.randn(H, generator=g)).to(dtype)
    total = res + delta.float()
    pick = torch.tensor([7, 0, 39] * 11, dtype=torch.int32)
    # float32: a sum of H squares in another order; bfloat16: one rounding of the result
    tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=1e-5)
    for d, rows in ((delta, None), (None, None), (delta, pick), (None, pick)):
        r = res.clone().cuda()
        out = torch.full((40 if rows is None else 33, H), float("nan"), dtype=dtype, device="cuda")
        ops.add_rmsnorm(r, None if d is None else d.cuda(), w.cuda(), 1e-6, out, None if rows is None else rows.cuda())
        x = (res if d is None else total).double()
        want = x / (x.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
        torch.testing.assert_close(out.cpu().double(), want if rows is None else want[rows.long()], **tol)
        assert torch.equal(r.cpu(), total if d is not None and rows is None else res)


@pytest.mark.parametrize("nq,nkv,hd,rot", [(14, 2, 64, 64), (28, 4, 128, 128), (6, 2, 128, 32)])
def test_rotation_does_not_depend_on_the_number_of_tokens(ops, nq, nkv, hd, rot):
    """One, two and four tokens a CTA (up to 592, 1,184 and more tokens): the same bits as in steps of 100."""
    T, g = 1189, torch.Generator().manual_seed(hd + rot)
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, generator=g).bfloat16().cuda()
    pos = torch.randint(0, 4000, (T,), generator=g, dtype=torch.int32).cuda()
    inv = (10000.0 ** (-torch.arange(0, rot, 2) / rot)).cuda()
    slots = torch.randperm(1200, generator=g)[:T].to(torch.int32).cuda()

    def run(cuts):
        x, k, v = qkv.clone(), *(torch.zeros(75, nkv, 16, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        for lo, hi in zip(cuts, cuts[1:]):
            ops.rope_store(x[lo:hi], pos[lo:hi].clone(), inv, nq, nkv, hd, rot, slots[lo:hi].clone(), k, v)
        return x, k, v
    want = run(list(range(0, T, 100)) + [T])
    for cuts in ([0, T], [0, 593, T], [0, 1185, T]):
        for a, b in zip(run(cuts), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("T", [33, 64])
@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (5, 1, 128), (40, 8, 128)])
def test_rotation_of_partial_sums_does_not_depend_on_the_number_of_tokens(ops, T, nq, nkv, hd):
    """Eight heads a CTA (33 tokens and more), the last CTA with fewer: the same bits as token by token."""
    g, W = torch.Generator().manual_seed(T + hd), (nq + 2 * nkv) * hd
    parts, bias = torch.randn(3, T, W, generator=g).cuda(), torch.randn(W, generator=g).bfloat16().cuda()
    pos = torch.arange(T, dtype=torch.int32).cuda()
    inv = (10000.0 ** (-torch.arange(0, hd, 2) / hd)).cuda()

    def run(steps):
        q = torch.zeros(T, W, dtype=torch.bfloat16, device="cuda")
        k, v = (torch.zeros(5, nkv, 16, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        for lo, hi in steps:
            ops.rope_store(q[lo:hi], pos[lo:hi].clone(), inv, nq, nkv, hd, hd, pos[lo:hi].clone(), k, v,
                           partials=parts[:, lo:hi].contiguous(), bias=bias)
        return q, k, v
    for a, b in zip(run([(0, T)]), run([(t, t + 1) for t in range(T)])):
        assert torch.equal(a, b)


@pytest.mark.parametrize("hd,page,window", [(64, 16, None), (128, 8, None), (128, 128, None), (64, 32, 300)])
def test_decode_merge_around_its_loads(ops, hd, page, window):
    """Requests of 1, 2, 15 to 17 and 31, 32 chunks of 128 keys: outputs are fetched 16 chunks at a time."""
    reqs = [(n, 1) for n in (0, 127, 128, 1919, 1920, 2047, 2048, 2175, 2176, 3967, 4090)]
    mgr, batch, qkv, view, _ = attention_case(ops, nq=6, nkv=2, hd=hd, page_size=page, window=window, requests=reqs,
                                              dtype=torch.bfloat16)
    out = torch.full((len(reqs), 6 * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    host, ref = batch_to_cpu(batch), torch.empty(len(reqs), 6 * hd, dtype=torch.bfloat16)
    ops.paged_attention(qkv, view.keys, view.values, batch, batch.groups[0], 6, 2, hd, hd ** -0.5, window, out,
                        storage=view.storage)
    ops.check_errors()
    HOST.paged_attention(qkv.cpu(), view.keys.cpu(), view.values.cpu(), host, host.groups[0], 6, 2, hd, hd ** -0.5,
                         window, ref)
    # (the bounds of the bfloat16 attention tests: probabilities and result are rounded to 2^-9 of themselves)
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=1.6e-2, atol=1e-2)
