"""Workspaces of the fused products: one per stream that grows, and one per stream capture."""
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


@pytest.mark.gpu
def test_a_captured_product_survives_growth_of_the_stream_workspace():
    """Two captures on one stream, the second with a larger layer, the allocator's cache emptied in between: the first
    graph still gives the eager product, on inputs it has not seen."""
    from alpaca_lora_4bit_b200 import quant_cuda, synth
    dev = torch.device("cuda")
    small, large = (synth.make_layer(K, N, 32, act_order=True, seed=K).to(dev) for K, N in ((512, 512), (4096, 2048)))
    xs = [synth.make_acts(300, L.qweight.shape[0] * 8, seed=3).to(dev) for L in (small, large)]
    outs = [torch.empty((300, L.qweight.shape[1]), dtype=torch.float16, device=dev) for L in (small, large)]
    stream, graphs = torch.cuda.Stream(), []

    def product(i):
        L = (small, large)[i]
        quant_cuda.gemm(xs[i], L.qweight, outs[i], L.scales, L.qzeros, L.g_idx)

    for i in (0, 1):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            if i:
                product(0)
            product(i)
        graphs.append(graph)
        torch.cuda.empty_cache()
    for x in xs:
        x.mul_(0.5)
    graphs[1].replay()
    graphs[0].replay()
    torch.cuda.synchronize()
    got = [o.clone() for o in outs]
    for i in (0, 1):
        product(i)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, outs)) and quant_cuda.device_status() == 0
