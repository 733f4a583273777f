"""Latent attention of prompt portions over expanded keys and values, against the same layer over the latents:
both in bfloat16 beside the float32 path, at the bounds of the tiles that are gathered."""

import pytest
import torch

from somi_inference_b200.config.spec import PartSpec
from somi_inference_b200.parts import MIXERS, BuildContext
from somi_inference_b200.parts.base import PagedKVNeeds
from tests.gpu_util import Steps

pytestmark = pytest.mark.gpu
HIDDEN, HEADS, RANK = 64, 6, 72


@pytest.fixture(scope="module")
def ops():
    from somi_inference_b200.ops import cuda_ops
    return cuda_ops()


def layers(ops, dim, window):
    names = ("q_down", "q_norm", "q_up", "k_up", "v_up", "sink", "out", "kv_down", "kv_norm")
    spec = PartSpec("latent_attention", {
        "hidden_size": HIDDEN, "heads": HEADS, "key_dim": dim, "value_dim": dim, "q_rank": 40, "kv_rank": RANK,
        "scale": 0.5 * dim ** -0.5, "window": window, "own_latent": True, "sink": True, "eps": 1e-5,
        "names": {n: n for n in names}})
    g = torch.Generator().manual_seed(dim)
    w = {d.name: (torch.randn(d.shape, generator=g) * (d.shape[-1] ** -0.5 if len(d.shape) > 1 else 1.0)).bfloat16()
         for d in MIXERS.declare(spec)}
    out = {}
    for dtype in (torch.bfloat16, torch.float32):
        ctx = BuildContext(dtype=dtype, device=torch.device("cuda"), ops=ops)
        out[dtype] = MIXERS.build(spec, {k: ctx.place(v, matrix=v.dim() > 1) for k, v in w.items()}, ctx)
    return out


ENDS = [{0: 127, 1: 128, 2: 129, 3: 300, 4: 385, 5: 5}, {0: 1, 1: 1, 2: 257, 3: 130, 4: 255, 5: 200}]
RUNS = [{0: 40, 1: 150, 2: 2, 3: 95, 4: 96, 5: 200}, {0: 300, 1: 1, 2: 97, 3: 20, 4: 130, 5: 1}]
LONG = [{0: 900, 1: 2}, {0: 1, 1: 96}]


@pytest.mark.parametrize("steps,expansions,most", [(ENDS, 2, None), (RUNS, 4, None), (LONG, 2, None), (ENDS, None, 3)])
@pytest.mark.parametrize("dim,window,page", [(64, None, 16), (128, None, 8), (64, 127, 32), (128, 300, 16), (64, 1, 16)])
def test_expanded_portions(ops, monkeypatch, dim, window, page, steps, expansions, most):
    """Two steps: portions that end around a tile of 128 positions, then portions and single tokens behind
    them (their first visible key in, on and behind a tile's first position); or portions of 96 rows and
    more between shorter ones, which read the latents; or a short prompt beside a long request; or a workspace
    of `most` tiles, so that portions go in several runs and one of more tiles reads the latents."""
    mixers = layers(ops, dim, window)
    if most:
        monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", most * 128 * 2 * (RANK + 2 * HEADS * dim))
    paged = PagedKVNeeds(1, RANK, window, value_dim=0)
    error, route = {}, []
    real = ops.latent_portions
    ops.latent_portions = lambda *a: (route.append(1), real(*a))[1]
    was = ops.use_expanded_latent
    try:
        caches = {key: Steps(ops, 6, paged=paged, page_size=page, max_len=1024, dtype=key[0], seed=3)
                  for key in ((torch.float32, False), (torch.bfloat16, False), (torch.bfloat16, True))}
        g = torch.Generator().manual_seed(1)
        for counts in steps:
            x = torch.randn(sum(counts.values()), HIDDEN, generator=g).bfloat16().cuda()
            got = {}
            for key, cache in caches.items():
                ops.use_expanded_latent = key[1]
                batch, _ = cache.step(counts)
                y = mixers[key[0]].forward(x.to(key[0]), batch, cache.mgr.view(0), True)
                got[key] = (y.double() if y.dim() == 2 else y.double().sum(0))
            want = got[torch.float32, False]
            for key in ((torch.bfloat16, False), (torch.bfloat16, True)):
                off = (got[key] - want).norm(dim=1) / want.norm(dim=1).mean()
                error.setdefault(key[1], []).append(off)
        ops.check_errors()
    finally:
        ops.latent_portions, ops.use_expanded_latent = real, was
    assert len(route) == expansions if expansions else len(route) >= 3
    # bfloat16 either way: an operand of each of the two per-head products is rounded to 2^-9 of itself
    for plain, expanded in zip(error[False], error[True]):
        assert expanded.mean() <= 1.3 * plain.mean() + 1e-4
        assert expanded.max() <= 2 * plain.max() + 1e-3


def test_short_portions_read_the_latents(ops):
    mixer = layers(ops, 64, None)[torch.bfloat16]
    cache = Steps(ops, 2, paged=PagedKVNeeds(1, RANK, None, value_dim=0), dtype=torch.bfloat16)
    batch, _ = cache.step({0: 95, 1: 40})
    args = (batch, batch.groups[0], cache.mgr.view(0).paged.keys, HEADS, RANK)
    assert not ops.latent_expands(*args, 64, 64, None, torch.bfloat16)
    batch, _ = cache.step({0: 2, 1: 96})
    args = (batch, batch.groups[0], cache.mgr.view(0).paged.keys, HEADS, RANK)
    assert ops.latent_expands(*args, 64, 64, None, torch.bfloat16)
    assert not ops.latent_expands(*args, 64, 128, None, torch.bfloat16)
    assert not ops.latent_expands(*args, 64, 64, None, torch.float32)
    assert mixer.kv_up.shape == (2 * HEADS * 64, RANK)
