"""The kernel table's host side (`ops/cuda.py`) without a GPU: what it hands to a launcher, and what it
refuses before it launches anything.  The library is a stand-in whose functions are called through ctypes."""

import ctypes
from types import SimpleNamespace

import pytest
import torch

from somi_inference_b200.ops import cuda
from somi_inference_b200.ops.build import build

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

    def call(decay=at, positions=at, freq=at, angles=at, rot=16):
        return lib.somi_matrix_state_chunks(at, at, at, L(256), L(256), L(256), I(0), F(1), decay, at, at, at, at, I(1), I(1),
                                            I(64), I(2), I(1), I(64), positions, freq, I(rot), angles, at, at, P(0))
    assert call(decay=P(0)) == call(decay=P(0), rot=0) == cuda.ERR_UNSUPPORTED
    assert call(positions=P(0)) == call(freq=P(0)) == call(angles=P(0)) == cuda.ERR_UNSUPPORTED


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
