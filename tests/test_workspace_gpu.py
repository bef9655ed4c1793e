"""Workspaces of captured products on the GPU."""
import pytest
import torch

from alpaca_lora_4bit_b200 import _lib, quant_cuda, synth
from tests.test_gemm_plan_cpu import CLUSTER, CUT, KERNEL, plan

pytestmark = pytest.mark.gpu


def _capture(stream, *products):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for p in products:
            p()
    return graph


def test_a_captured_product_survives_growth_of_the_stream_workspace():
    """Two captures on one stream, the second with a larger layer, the allocator's cache emptied in between: the first
    graph still gives the eager product, on inputs it has not seen.  Both layers exchange sums through the workspace."""
    dev, M = torch.device("cuda"), 40
    layers = [synth.make_layer(K, N, 128, act_order=True, seed=K).to(dev) for K, N in ((4096, 11008), (5120, 13824))]
    need = []
    for L in layers:
        K, N, G = L.qweight.shape[0] * 8, L.qweight.shape[1], L.scales.shape[0]
        p = plan(M, K, N, G, True, resident=None)
        assert p[KERNEL] == 4 and p[CUT] and p[CLUSTER] == 1, p
        need.append(int(_lib.lib().q4_gemm_workspace_bytes(K, N, G)))
    assert need[1] > need[0]
    xs = [synth.make_acts(M, L.qweight.shape[0] * 8, seed=3).to(dev) for L in layers]
    outs = [torch.empty((M, L.qweight.shape[1]), dtype=torch.float16, device=dev) for L in layers]
    stream, graphs = torch.cuda.Stream(), []

    def product(i):
        L = layers[i]
        quant_cuda.gemm(xs[i], L.qweight, outs[i], L.scales, L.qzeros, L.g_idx)

    for i in (0, 1):
        graphs.append(_capture(stream, *(lambda j=j: product(j) for j in range(i + 1))))
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


@pytest.mark.parametrize("M,act_order", [(1, False), (7, False), (1, True), (16, True)])
def test_captured_decode_has_a_workspace_of_its_own(M, act_order):
    """Graphs captured on a stream that has run no decode product before, the second replayed first, then both, then eager
    calls on the stream of the capture: the products of an eager call each time."""
    dev = torch.device("cuda")
    layers = [synth.make_layer(K, N, 128, act_order=act_order, seed=K + N).to(dev) for K, N in ((4096, 4096), (5120, 13824), (13824, 5120))]
    xs = [synth.make_acts(M, L.qweight.shape[0] * 8, seed=4).to(dev) for L in layers]
    stream = torch.cuda.Stream()

    def run(store):
        for i, L in enumerate(layers):
            quant_cuda.gemv(xs[i], L.qweight, store[i], L.scales, L.qzeros, L.g_idx if act_order else None, 128,
                            _lib.GEMV_ACT_ORDER if act_order else 0)

    def empty():
        return [torch.empty((M, L.qweight.shape[1]), dtype=torch.float16, device=dev) for L in layers]

    want, first, second, eager = empty(), empty(), empty(), empty()
    run(want)
    torch.cuda.synchronize()
    graphs = [_capture(stream, lambda o=o: run(o)) for o in (first, second)]
    assert _lib._capture_workspaces
    graphs[1].replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(second, want))
    for o in first + second:
        o.fill_(0)
    for g in graphs:                                     # one after the other: CTAs of a product wait for one another
        g.replay()
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(first + second, want + want))
    with torch.cuda.stream(stream):
        run(eager)
    torch.cuda.synchronize()
    assert not _lib._capture_workspaces
    assert all(torch.equal(a, b) for a, b in zip(eager, want)) and quant_cuda.device_status() == 0


@pytest.mark.parametrize("nbytes", [16, 4096, 65536, 131072, (1 << 20) + 16])
def test_clear(nbytes):
    buf = torch.full((nbytes + 64,), 7, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().q4_clear(buf.data_ptr() + 32, nbytes, torch.cuda.current_stream().cuda_stream), "clear")
    assert int(buf[32:32 + nbytes].sum()) == 0 and bool((buf[:32] == 7).all()) and bool((buf[32 + nbytes:] == 7).all())
