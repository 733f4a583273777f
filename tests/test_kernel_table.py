"""The kernel table's host side (`ops/cuda.py`) without a GPU: what it hands to a launcher, and what it
refuses before it launches anything.  The library is a stand-in whose functions are called through ctypes."""

import ctypes

import pytest
import torch

from somi_inference_b200.ops import cuda

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
