"""Scratch buffers: one per stream and tag, so that kernels of two streams never meet in one.  The CUDA calls are stood in for:
which buffer a call is handed is host work."""
import contextlib
import types

import pytest
import torch

from bamboo_b200 import layers, lib


@pytest.fixture
def streams(monkeypatch):
    """`.current`: raw handle of the current stream; `.allocated_on`: the stream of each allocation."""
    st = types.SimpleNamespace(current=100, allocated_on=[])
    empty = torch.empty

    @contextlib.contextmanager
    def on(stream):
        before, st.current = st.current, stream
        yield
        st.current = before

    def allocate(n, dtype=None, device=None):
        st.allocated_on.append(st.current)
        return empty(n, dtype=dtype)
    monkeypatch.setattr(lib, "_workspaces", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda dev: st.current)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda raw, device=None: raw)
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch, "empty", allocate)
    return st


def test_a_buffer_belongs_to_one_stream(streams):
    a = lib.workspace(100, "t")
    assert lib.workspace(50, "t") is a and lib.workspace(50, "t", stream=100) is a
    assert lib.workspace(100, "u") is not a
    b = lib.workspace(100, "t", stream=7)
    assert b is not a and b.data_ptr() != a.data_ptr()
    streams.current = 7
    assert lib.workspace(100, "t") is b
    # a larger one is allocated on the stream that uses it, like the first
    big = lib.workspace(4 << 20, "t", stream=100)
    assert big.numel() == 4 << 20 and lib.workspace(1, "t") is b
    assert streams.allocated_on == [100, 100, 7, 100]


def test_bias_gradients_in_line_and_beside_have_scratch_of_their_own(streams, monkeypatch):
    calls = []
    native = types.SimpleNamespace(bb_colsum_workspace_bytes=lambda rows, n: 4 * rows.value * n.value,
                                   bb_colsum_accum=lambda dy, ld, out, ws, *rest: calls.append((ws.value, rest[-1].value)) or 0)
    monkeypatch.setattr(lib, "load", lambda: native)
    monkeypatch.setattr(lib, "gemm", lambda *a, **k: None)
    monkeypatch.setattr(lib, "_stream", lambda raw=None: types.SimpleNamespace(value=streams.current if raw is None else raw))
    w, b = torch.nn.Parameter(torch.zeros(8, 8)), torch.nn.Parameter(torch.zeros(8))
    w.main_grad, b.main_grad = torch.zeros(8, 8), torch.zeros(8)
    dy = torch.zeros(128, 8, dtype=torch.bfloat16)
    layers._wgrad(dy, dy, w, b, stream=7)
    layers._wgrad(dy, dy, w, b)
    layers._wgrad(dy, dy, w, b, stream=7)
    assert [s for _, s in calls] == [7, 100, 7]
    assert calls[0][0] == calls[2][0] != calls[1][0]
