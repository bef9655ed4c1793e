"""Workspaces of decode and fused products: one per stream (the fused one grows), and a capture's own."""
import gc
import weakref

import pytest
import torch

from alpaca_lora_4bit_b200 import _lib

CPU, STREAM = torch.device("cpu"), 7


@pytest.fixture
def capture(monkeypatch):
    state = {"id": 0}
    monkeypatch.setattr(_lib, "_gemm_workspaces", {})
    monkeypatch.setattr(_lib, "_capture_workspaces", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["id"] > 0)
    monkeypatch.setattr(_lib, "capture_id", lambda stream: state["id"])
    return state


def test_a_capture_never_holds_a_workspace_that_growth_replaces(capture):
    """A graph replays with the addresses it was captured with.  Captured on a stream whose workspace a larger layer then
    replaced - in a later capture, or in the same one - it went on using freed memory."""
    mib = 1 << 20
    eager = _lib.gemm_workspace_for(CPU, STREAM, 30 * mib)
    capture["id"] = 1
    first = _lib.gemm_workspace_for(CPU, STREAM, 30 * mib)
    assert first.data_ptr() != eager.data_ptr() and _lib.gemm_workspace_for(CPU, STREAM, 25 * mib) is first
    assert int(first[:_lib._GEMM_WS_HEAD].sum()) == 0
    grown = _lib.gemm_workspace_for(CPU, STREAM, 40 * mib)
    assert grown.numel() >= 40 * mib and grown is not first
    assert any(w is first for w in _lib._capture_workspaces[(CPU.index, STREAM)][1])      # alive while the capture goes on
    capture["id"] = 2
    second = _lib.gemm_workspace_for(CPU, STREAM, 30 * mib)
    assert second is not first and second is not grown
    capture["id"] = 0
    assert _lib.gemm_workspace_for(CPU, STREAM, 30 * mib) is eager
    assert _lib.gemm_workspace_for(CPU, STREAM, 50 * mib) is not eager


def test_a_capture_has_a_decode_workspace_of_its_own(capture, monkeypatch):
    """First asked for inside a capture, the decode workspace was cleared by that graph's replay alone and then kept for the
    stream: later captures and eager calls on it counted arrivals in memory that nothing had cleared."""
    monkeypatch.setattr(_lib, "_workspaces", {})
    capture["id"] = 1
    first = _lib.workspace_for(CPU, STREAM)
    assert first.numel() == _lib._WS_BYTES and int(first[:_lib._DECODE_WS_HEAD].sum()) == 0
    assert _lib.workspace_for(CPU, STREAM) is first and not _lib._workspaces
    fused = _lib.gemm_workspace_for(CPU, STREAM, 1)
    assert fused is not first and _lib.workspace_for(CPU, STREAM) is first
    capture["id"] = 2
    second = _lib.workspace_for(CPU, STREAM)
    assert second is not first and int(second[:_lib._DECODE_WS_HEAD].sum()) == 0
    capture["id"] = 0
    eager = _lib.workspace_for(CPU, STREAM)
    assert eager is not first and eager is not second and int(eager.sum()) == 0 and _lib.workspace_for(CPU, STREAM) is eager
    capture["id"] = 3
    assert _lib.workspace_for(CPU, STREAM) is not eager


@pytest.mark.parametrize("ask", [lambda: _lib.workspace_for(CPU, STREAM), lambda: _lib.gemm_workspace_for(CPU, STREAM, 1)])
def test_what_a_capture_held_is_let_go_by_the_next_eager_call(capture, monkeypatch, ask):
    """... so that the memory goes with its graph.  (The last capture's workspaces of every stream stayed for good.)"""
    monkeypatch.setattr(_lib, "_workspaces", {})
    capture["id"] = 1
    kept = [weakref.ref(_lib.workspace_for(CPU, STREAM)), weakref.ref(_lib.gemm_workspace_for(CPU, STREAM + 1, 1))]
    assert all(r() is not None for r in kept)
    capture["id"] = 0
    ask()
    gc.collect()
    assert all(r() is None for r in kept)
