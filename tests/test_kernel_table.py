"""The kernel table's host side (`ops/cuda.py`) without a GPU: what it hands to a launcher, and what it
refuses before it launches anything.  The library is a stand-in whose functions are called through ctypes."""

import ctypes
import random
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from somi_inference_b200.config.spec import PartSpec
from somi_inference_b200.ops import cuda
from somi_inference_b200.ops.build import build
from somi_inference_b200.parts import MIXERS, BuildContext, Decoder

P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float


@pytest.fixture
def ops(monkeypatch):
    """A kernel table on CPU tensors with no library behind it yet."""
    monkeypatch.setattr(cuda, "_check", lambda *tensors: None)
    table = cuda.CudaOps.__new__(cuda.CudaOps)
    table.lib, table.launches = type("Library", (), {})(), 0
    table._q_maps, table._gemm_maps, table._tensor_maps = {}, {}, {}
    table._stream = lambda: P(0)
    return table


def test_maps_stay_alive_until_their_launch_returns(ops):
    """A launch with two tensor maps that both are new, often enough that the table of maps gets full between
    them: each address that arrives still holds what was written there."""
    bad, launches, churn, kept = [], [], [], [0]

    def make(at, tensor, rows, columns, box):
        ctypes.memmove(at, tensor.to_bytes(8, "little") * 16, 128)
        return 0

    def launch(w_map, x_map, box, M, N, K, *rest):
        launches.append((w_map, x_map))
        if len(ops._gemm_maps) < kept[0]:                             # take over what has been freed
            churn.extend((ctypes.c_ubyte * 256)() for _ in range(20000))
        kept[0] = len(ops._gemm_maps)
        for at, tensor in ((w_map, w.data_ptr()), (x_map, x.data_ptr())):
            if ctypes.string_at(at, 128) != tensor.to_bytes(8, "little") * 16:
                bad.append(len(launches))
        return 0
    ops.lib.somi_make_gemm_tensor_map = ctypes.CFUNCTYPE(I, P, P, L, L, I)(make)
    ops.lib.somi_skinny_gemm = ctypes.CFUNCTYPE(I, P, P, I, I, I, I, I, I, P, I, P, F, F, F, F, I, P)(launch)
    ops._gated = lambda gated: (F(0),) * 4
    store = torch.zeros(2 * 4200, 8, dtype=torch.bfloat16)
    for i in range(4200):
        w, x = store[2 * i:2 * i + 1], store[2 * i + 1:2 * i + 2]
        ops.skinny_gemm(x, w)
    assert len(launches) == 4200 and churn and not bad


class OnDevice(torch.Tensor):
    """A CPU tensor that the host side takes for one of the device's."""
    is_cuda = True


def on_device(*shape, dtype=torch.float32):
    return torch.zeros(*shape, dtype=dtype).as_subclass(OnDevice)


def test_a_recurrence_without_a_decay_is_refused(ops):
    """Neither a decay per head nor decay logits, whichever way the rows would go: portions in chunks, short
    portions, single tokens."""
    launches = []
    for name in ("somi_matrix_state_chunks", "somi_matrix_state_prepare", "somi_matrix_state_scan"):
        setattr(ops.lib, name, lambda *args: launches.append(args) or 0)
    ops.use_scan_chunks, ops.prefill_q_tile = True, 64
    H, d, T = 2, 64, 80
    for n_portions in (1, 0):
        batch = SimpleNamespace(num_tokens=T, num_requests=1, num_prefill_requests=n_portions, max_q_len=T,
                                num_prefill_tokens=T * n_portions, cu_q=on_device(2), state_slot=on_device(1),
                                tiles={64: torch.zeros(2 * n_portions, 3)})
        qkv, state, y = on_device(T, 3 * H * d, dtype=torch.bfloat16), on_device(1, H, d, d), on_device(T, H * d)
        with pytest.raises(cuda.KernelError, match="decay"):
            ops.matrix_state_scan(qkv[:, :H * d], qkv[:, H * d:2 * H * d], qkv[:, 2 * H * d:], state, batch, y, H, H, d, d)
    assert not launches


def test_the_chunks_launcher_refuses_null_arguments():
    """A launcher's checks come before its first launch, so they are the same without a device."""
    lib = ctypes.CDLL(build(verbose=False))
    at = P(1 << 16)

    def call(decay=at, positions=at, freq=at, angles=at, rot=16, y=at):
        return lib.somi_matrix_state_chunks(at, at, at, L(256), L(256), L(256), I(0), F(1), decay, at, at, at, at, I(1), I(1),
                                            I(64), I(2), I(1), I(64), positions, freq, I(rot), angles, at, y, I(0), P(0))
    assert call(decay=P(0)) == call(decay=P(0), rot=0) == cuda.ERR_UNSUPPORTED
    assert call(positions=P(0)) == call(freq=P(0)) == call(angles=P(0)) == cuda.ERR_UNSUPPORTED
    assert call(y=P((1 << 16) + 4)) == cuda.ERR_UNSUPPORTED          # (rows are stored 16 bytes at a time)


@pytest.mark.parametrize("n,nq,nkv,hd,positions,window", [(64, 40, 8, 128, 32768, None), (64, 40, 8, 128, 32768, 1024),
                                                          (3, 14, 2, 64, 512, None), (3, 14, 2, 64, 131072, 65)])
def test_scratch_of_float32_single_tokens_is_bounded(ops, monkeypatch, n, nq, nkv, hd, positions, window):
    """Every request is in one launch, no launch's partial results take more than 128 MB, and a window needs
    only the chunks that it meets."""
    calls, sizes = [], []
    ops.lib.somi_attention_f32_supported = lambda *args: 1
    ops.lib.somi_attention_f32_single = lambda *args: calls.append([getattr(a, "value", a) for a in args]) or 0
    ops.use_f32_attention, ops.f32_chunk, ops.prefill_q_tile, ops.generic_q_tile = True, 64, 64, 16
    kv = on_device(1, nkv, 16, hd)
    group = SimpleNamespace(block_table=on_device(1, 1), width=positions // 16)
    batch = SimpleNamespace(num_requests=n + 2, num_prefill_requests=2, num_prefill_tokens=70, cu_q=on_device(1),
                            ctx_len=on_device(1), tiles={64: torch.zeros(0, 3), 16: torch.zeros(0, 3)})
    real = torch.empty
    monkeypatch.setattr(cuda.torch, "empty", lambda size, **kw: sizes.append(size) or real(1, **kw))
    ops.paged_attention(on_device(1, (nq + 2 * nkv) * hd), kv, kv, batch, group, nq, nkv, hd, 1.0, window, on_device(1, nq * hd))
    chunks = -(-positions // 64) if window is None else max((p + window - 1) // 64 - p // 64 + 1 for p in range(64))
    at = 0
    for row, request, count, most in ((c[2], c[3], c[4], c[-3]) for c in calls):
        assert (row, request, most) == (70 + at, 2 + at, chunks)
        assert count * nq * chunks * (hd + 2) <= sizes[0] <= (1 << 25)
        at += count
    assert at == n and len(sizes) == 1


def portions(*lengths, singles=()):
    """A step of portions (cached tokens, tokens) and single tokens behind them, as the kernel table reads it."""
    reqs = [*lengths, *((c, 1) for c in singles)]
    cu = np.cumsum([0] + [q for _, q in reqs])
    T, widest = int(cu[-1]), max(c + q for c, q in reqs)
    tiles = {t: torch.tensor([(r, cu[r] + i, min(t, q - i)) for r, (_, q) in enumerate(lengths) for i in range(0, q, t)],
                             dtype=torch.int32).view(-1, 3) for t in (16, 64, 128, 256)}
    return SimpleNamespace(
        num_tokens=T, num_requests=len(reqs), num_prefill_requests=len(lengths), num_prefill_tokens=int(cu[len(lengths)]),
        max_q_len=max(q for _, q in reqs), cu_q=on_device(len(reqs) + 1), ctx_len=on_device(len(reqs)),
        state_slot=on_device(len(reqs)), positions=on_device(T, dtype=torch.int32), tiles=tiles,
        groups=[SimpleNamespace(block_table=on_device(len(reqs), 1), width=-(-widest // 16))],
        host=SimpleNamespace(cu_q=cu, ctx_len=np.array([c for c, _ in reqs]), plans={}))


@pytest.fixture
def latents(ops):
    """The kernel table with stand-ins behind latent attention; `calls` names them with their numbers."""
    ops.calls = []
    for name in ("somi_latent_gather", "somi_attention_prefill_pp_columns", "somi_latent_attention_mma"):
        setattr(ops.lib, name, lambda *args, name=name: ops.calls.append((name, [getattr(a, "value", a) for a in args])) or 0)
    ops.lib.somi_prefill_pp_supported = ops.lib.somi_latent_attention_mma_supported = lambda *args: 1
    ops.lib.somi_latent_attention_splits = lambda *args: 1
    ops._q_tensor_map = lambda t: P(0)
    ops.use_expanded_latent, ops.use_mma_latent = True, True
    ops.latent_tile, ops.prefill_pp_q_tile, ops.latent_q_tile = 128, 256, 16
    return ops


def expanded_tiles(ops, batch, window=None, heads=1, rank=8, dim=64):
    """Tiles that each product over expanded latents runs over."""
    T = batch.num_tokens
    q, out = (on_device(T, heads * dim, dtype=torch.bfloat16) for _ in range(2))
    ops.calls.clear()
    for run in ops.latent_runs(batch, window, heads, rank, dim):
        if run[2]:
            ops.latent_portions(q, on_device(1, 1, 16, rank, dtype=torch.bfloat16),
                                on_device(2 * heads * dim, rank, dtype=torch.bfloat16), batch, batch.groups[0], heads,
                                rank, dim, 1.0, window, None, out, run)
    return [args[10] for name, args in ops.calls if name == "somi_latent_gather"]


def test_expanded_positions_are_the_portions_own(latents):
    """A prompt beside a long request expands its own positions; other lengths that round to the same
    number give the same launches, and no number is short."""
    assert expanded_tiles(latents, portions((0, 96), singles=(16000,))) == [1]
    assert expanded_tiles(latents, portions((3000, 100), singles=(16000,)), window=128) == [3]
    rng = random.Random(1)
    for _ in range(300):
        reqs = [(rng.randrange(0, 3000), rng.randrange(96, 700)) for _ in range(rng.randrange(1, 6))]
        window = rng.choice((None, 1, 127, 128, 129, 1000))
        read = sum(len({p // 128 for p in range(0 if window is None else max(0, c - window + 1), c + q)}) for c, q in reqs)
        (tiles,) = expanded_tiles(latents, portions(*reqs, singles=(9000,)), window)
        assert read <= tiles <= 1.25 * read
    assert len({expanded_tiles(latents, portions((0, q)))[0] for q in range(96, 8192, 32)}) <= 24


@pytest.mark.parametrize("window", [None, 300])
def test_a_portion_goes_its_own_way_whatever_else_is_in_the_step(latents, window):
    """Latent attention: whether a portion reads expanded keys and values follows from its rows and positions; the
    runs go through all requests in order, and each launch reaches its run's tiles and rows."""
    rng = random.Random(2)
    sizes = [(0, 95), (0, 96), (0, 40), (500, 300), (0, 2), (40000, 200), (20000, 96)]
    heads, rank, dim = 28, 512, 128
    position = 2 * (rank + 2 * heads * dim)              # bytes

    def alone(size):
        return latents.latent_runs(portions(size), window, heads, rank, dim)[0][2] > 0
    assert [alone(s) for s in sizes] == [False, True, False, True, False, window is not None, True]
    for _ in range(100):
        reqs = [rng.choice(sizes) for _ in range(rng.randrange(1, 7))]
        batch = portions(*reqs, singles=rng.choice(((), (7, 9000))))
        runs = latents.latent_runs(batch, window, heads, rank, dim)
        assert [r for a, b, _ in runs for r in range(a, b)] == list(range(batch.num_requests))
        for a, b, tiles in runs:
            assert all(r < len(reqs) and alone(reqs[r]) if tiles else r >= len(reqs) or not alone(reqs[r]) for r in range(a, b))
            assert 0 <= tiles * 128 * position <= 1 << 29
            at, n = latents._tiles_of(batch, 64, a, b)
            mine = [t for t in batch.tiles[64].tolist() if a <= t[0] < b]
            assert n == len(mine) and (not n or batch.tiles[64][(at.value - batch.tiles[64].data_ptr()) // 12].tolist() == mine[0])


@pytest.mark.parametrize("heads,dim", [(128, 128), (16, 64)])
def test_the_workspace_of_expanded_latents_is_bounded_in_bytes(latents, monkeypatch, heads, dim):
    """Many heads expand fewer positions side by side: no workspace takes more than 512 MB."""
    rank, real, sizes = 512, torch.empty, []
    monkeypatch.setattr(cuda.torch, "empty", lambda size, **kw: sizes.append(size) or real(1, **kw))
    monkeypatch.setattr(cuda.torch.nn.functional, "linear", lambda x, w: torch.zeros(1, 1, dtype=torch.bfloat16))
    batch = portions(*((3000, 500),) * 12, (30000, 100))
    expanded_tiles(latents, batch, None, heads, rank, dim)
    rows = [s[0] for s in sizes if s[1] == rank]
    assert rows and all(r * (rank + 2 * heads * dim) * 2 <= 1 << 29 for r in rows)


def latent_layer(ops, windows, dim=64):
    """The last of a model's latent layers, one per window, and the context that they were built in."""
    ops.check_latent_geometry = lambda *args: None
    names = ("q_down", "q_norm", "q_up", "k_up", "v_up", "out", "kv_down", "kv_norm")
    ctx = BuildContext(dtype=torch.bfloat16, device=torch.device("cpu"), ops=ops)
    for window in windows:
        spec = PartSpec("latent_attention", {
            "hidden_size": 64, "heads": 2, "key_dim": dim, "value_dim": dim, "q_rank": 8, "kv_rank": 8, "scale": 1.0,
            "window": window, "own_latent": True, "eps": 1e-5, "names": {n: n for n in names}})
        mixer = MIXERS.build(spec, {d.name: torch.ones(d.shape, dtype=torch.bfloat16) for d in MIXERS.declare(spec)}, ctx)
    return mixer, ctx


def test_expansion_weights_are_held_where_they_are_read(latents):
    """Sizes that never read expanded keys and values hold no matrix for them; where they do, W_uv lies in
    memory once."""
    latents.lib.somi_prefill_pp_supported = lambda nq, nkv, hd, page: hd.value in (64, 128)
    mixer, ctx = latent_layer(latents, [None], dim=32)
    assert mixer.kv_up is None and not ctx.layout_facts
    mixer, _ = latent_layer(latents, [None])
    assert mixer.kv_up.shape == (2 * 2 * 64, 8) and mixer.v_up.shape == (2, 64, 8)
    assert mixer.v_up.data_ptr() == mixer.kv_up[2 * 64:].data_ptr()


def test_the_number_of_expanded_tiles_is_a_fact_of_the_layout(latents):
    """Two steps of equal sizes whose portions read another number of tiles are told apart; layers that are
    alike enter one fact."""
    _, ctx = latent_layer(latents, (None, None, 256))
    model = SimpleNamespace(ctx=ctx)
    facts = [Decoder.layout_facts(model, portions((c, 100), singles=(5000,))) for c in (0, 28, 29, 2000)]
    assert len(facts[0]) == 2 and facts[0] == facts[1] and len(set(facts)) == 3
    assert Decoder.layout_facts(model, portions(singles=(5000,))) == ()
    # equal numbers of rows and tiles, but the run of short portions is at other rows
    a, b = portions((0, 110), (0, 60)), portions((0, 112), (0, 58))
    assert all(a.tiles[t].shape == b.tiles[t].shape for t in a.tiles) and a.num_tokens == b.num_tokens
    assert Decoder.layout_facts(model, a) != Decoder.layout_facts(model, b)


def test_a_portion_goes_through_the_recurrence_its_own_way(ops):
    """In chunks or step by step by its own rows; the launches cover all requests in order, with their rows."""
    calls = []
    for name in ("chunks", "prepare", "scan"):
        setattr(ops.lib, f"somi_matrix_state_{name}",
                lambda *args, name=name: calls.append((name, [getattr(a, "value", a) for a in args])) or 0)
    ops.use_scan_chunks, ops.prefill_q_tile = True, 64
    H, d, rng = 2, 64, random.Random(3)
    least = int(ops.SCAN_CHUNK_ROWS * d)
    for _ in range(100):
        lengths = [rng.choice((2, 17, least - 1, least, least + 1, 5 * least)) for _ in range(rng.randrange(1, 6))]
        batch = portions(*((0, n) for n in lengths), singles=rng.choice(((), (5, 9))))
        T, R = batch.num_tokens, batch.num_requests
        qkv = on_device(T, 3 * H * d, dtype=torch.bfloat16)
        calls.clear()
        ops.matrix_state_scan(qkv[:, :H * d], qkv[:, H * d:2 * H * d], qkv[:, 2 * H * d:], on_device(R, H, d, d), batch,
                              on_device(T, H * d), H, H, d, d, decay=on_device(H))
        at, cu = 0, batch.cu_q.data_ptr()
        for name, args in calls:
            if name == "prepare":
                continue
            n = args[14] if name == "chunks" else args[-10]
            first = ((args[10] if name == "chunks" else args[-13]) - cu) // 4
            assert first == at and n >= 1
            for r in range(at, at + n):
                assert (r < len(lengths) and lengths[r] >= least) == (name == "chunks")
            if name == "chunks":
                assert args[13] == sum(-(-q // 64) for q in lengths[at:at + n]) and args[15] == batch.host.cu_q[at + n]
            at += n
        assert at == R


def test_the_chunks_workspace_is_bounded(ops):
    """Portions whose chunks' states together take more than 512 MB go one run behind the other, one that
    takes more by itself step by step."""
    heads, d = 28, 128
    runs = ops.scan_runs(portions((0, 10000), (0, 10000), (0, 20000), singles=(4,)), heads, d)
    assert runs == ((0, 1, 157), (1, 2, 157), (2, 4, 0))
    assert all(n * heads * d * d * 4 <= 1 << 29 for _, _, n in runs)


def test_the_chunks_workspace_has_a_place_for_every_chunk(ops, monkeypatch):
    """The states' scratch is one per chunk of 128 rows, at most one more a request; the kernels' places in it ((rows in front + 127 r) / 128 for
    request r's first chunk) are each a chunk's own and lie inside."""
    sizes, calls, heads, d, rng = [], [], 2, 64, random.Random(5)
    ops.lib.somi_matrix_state_chunks = lambda *args: calls.append([getattr(a, "value", a) for a in args]) or 0
    ops.use_scan_chunks, ops.prefill_q_tile = True, 64
    real = torch.empty
    monkeypatch.setattr(cuda.torch, "empty", lambda size, **kw: sizes.append(size) or real(1, **kw))
    for _ in range(200):
        lengths = [rng.choice((96, 97, 127, 128, 129, 192, 193, 256, 257, rng.randrange(96, 2000))) for _ in range(rng.randrange(1, 9))]
        batch = portions(*((0, n) for n in lengths))
        qkv = on_device(batch.num_tokens, 3 * heads * d, dtype=torch.bfloat16)
        sizes.clear(), calls.clear()
        ops.matrix_state_scan(qkv[:, :heads * d], qkv[:, heads * d:2 * heads * d], qkv[:, 2 * heads * d:], on_device(len(lengths), heads, d, d),
                              batch, on_device(batch.num_tokens, heads * d), heads, heads, d, d, decay=on_device(heads))
        chunks = [-(-n // 128) for n in lengths]
        assert len(sizes) == len(calls) == 1 and sizes[0] <= (sum(chunks) + len(lengths)) * heads * d * d
        starts = [(sum(lengths[:r]) + 127 * r) // 128 for r in range(len(lengths))]
        places = [s + c for s, n in zip(starts, chunks) for c in range(n)]
        assert len(set(places)) == len(places) and (max(places) + 1) * heads * d * d <= sizes[0]
