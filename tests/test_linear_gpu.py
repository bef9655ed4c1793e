"""The no-grad forward of the quant linear module through the native call: bias and residual in the kernels'
epilogues, every row range and layer format, against the oracle's reconstruct."""
import pytest
import torch

from alpaca_lora_4bit_b200 import autograd_4bit as a4, matmul_utils_4bit as mm4b, quant_cuda, synth
from oracle import q4_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
K, N = 512, 768


def build(fmt, groupsize):
    layer = synth.make_layer(K, N, groupsize, act_order=fmt == "act", seed=3)
    mod = a4.Autograd4bitQuantLinear(K, N, groupsize=-1 if fmt == "v1" else groupsize, is_v1_model=fmt == "v1")
    gen = torch.Generator().manual_seed(4)
    bias = torch.randn(N, generator=gen).half()
    if fmt == "v1":
        scales = (torch.rand(N, 1, generator=gen) * 0.018 + 0.002).half()
        zeros = (scales.float() * torch.randint(1, 16, (N, 1), generator=gen)).half()
        mod.scales, mod.zeros = scales.to(DEV), zeros.to(DEV)
        w = orc.recons_v1(layer.qweight, scales.reshape(-1), zeros.reshape(-1))
    else:
        mod.scales, mod.qzeros, mod.g_idx = layer.scales.to(DEV), layer.qzeros.to(DEV), layer.g_idx.to(DEV)
        w = orc.recons_v2(layer.qweight, layer.scales, layer.qzeros, layer.g_idx)
    mod.qweight, mod.bias = layer.qweight.to(DEV), bias.to(DEV)
    return mod.eval(), w.float(), bias.float()


@pytest.mark.parametrize("rows", [1, 2, 8, 9, 16, 17, 33, 129, 300])
@pytest.mark.parametrize("fmt,groupsize", [("seq", 128), ("seq", 32), ("act", 128), ("v1", 512)])
def test_module_without_grad_adds_bias_and_residual(fmt, groupsize, rows):
    mod, w, bias = build(fmt, groupsize)
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, K, generator=gen).half()
    res = torch.randn(rows, N, generator=gen).half()
    mm4b.act_order = fmt == "act"
    try:
        with torch.no_grad():
            y = mod(x.to(DEV))
            y3 = mod(x.to(DEV).reshape(1, rows, K))
            mod.offer_residual(res.to(DEV))
            yr = mod(x.to(DEV))
            mod.disable_bias = True
            yn = mod(x.to(DEV))
    finally:
        mm4b.act_order = False
    torch.cuda.synchronize()
    want = x.float() @ w
    for got, ref in ((y, want + bias), (yr, want + bias + res.float()), (yn, want)):
        # fp16 result of sums in fp32; decode kernels work on the exact weights, the reference on their fp16 rounding
        assert float((got.float().cpu() - ref).norm() / ref.norm()) <= 2e-3
    assert y3.shape == (1, rows, N) and torch.equal(y3.reshape(rows, N), y)
    assert quant_cuda.device_status() == 0


def test_native_call_leaves_operands_it_does_not_take():
    mod, w, bias = build("seq", 128)
    x = torch.randn(4, K, generator=torch.Generator().manual_seed(1))
    ref = x @ w + bias
    with torch.no_grad():
        for xx in (x.half().to(DEV).t().contiguous().t(), x.to(DEV), x.bfloat16().to(DEV)):     # not contiguous, fp32, bf16
            y = mod(xx)
            assert float((y.float().cpu() - ref).norm() / ref.norm()) <= 1e-2 and y.shape == (4, N)
        assert mod(x[:0].half().to(DEV)).shape == (0, N)
        with pytest.raises((RuntimeError, AssertionError)):
            mod(torch.zeros(4, K + 128, dtype=torch.float16, device=DEV))


@pytest.mark.parametrize("K2,N2", [(128, 256), (256, 128), (512, 768), (640, 384), (2048, 5120), (11008, 512)])
@pytest.mark.parametrize("rows", [9, 17, 129, 257, 700])
def test_first_format_large_products_both_ways(K2, N2, rows):
    """Layers of the first format above the switch threshold: the fused kernels (output columns a multiple of 256) and
    the reconstruct path (the rest) against fp32 products of the same fp16 weights, and the gradient the transpose."""
    gen = torch.Generator().manual_seed(K2 + rows)
    qweight = torch.randint(-2 ** 31, 2 ** 31 - 1, (K2 // 8, N2), generator=gen).to(torch.int32).to(DEV)
    scales = (torch.rand(N2, 1, generator=gen) * 0.018 + 0.002).half()
    scales[::7] = -3.25 * scales[::7]                       # negative scales, and with the next line some above 2
    scales[3::31] = 2.5
    zeros = (scales.float() * torch.randint(1, 16, (N2, 1), generator=gen)).half().to(DEV)
    scales = scales.to(DEV)
    bias = torch.randn(N2, generator=gen).half().to(DEV)
    w = torch.empty((K2, N2), dtype=torch.float16, device=DEV)
    quant_cuda.vecquant4recons_v1(qweight, w, scales.reshape(-1), zeros.reshape(-1))
    x = torch.randn(2, rows, K2, generator=gen).half().to(DEV)[1:].requires_grad_(True)
    dy = torch.randn(1, rows, N2, generator=gen).half().to(DEV)
    res = torch.randn(1, rows, N2, generator=gen).half().to(DEV)
    y = a4.AutogradMatmul4bitCuda.apply(x, qweight, scales, zeros, None, 4, 15, bias, res)
    (dx,) = torch.autograd.grad(y, [x], dy)
    want = (x.detach().double() @ w.double() + bias.double()) + res.double()
    dwant = dy.double() @ w.double().t()
    for got, ref in ((y, want), (dx, dwant)):                # fp32 sums rounded to fp16 (twice: product, residual): 2 * 2^-11
        assert got.shape == ref.shape and float((got.double() - ref).norm() / ref.norm()) <= 1e-3
    with torch.no_grad():
        y2 = mm4b.linear(x, qweight, scales, zeros, None, K2, bias, res)
        yt = torch.func.vmap(lambda v: mm4b.matmul4bit(v, qweight, scales, zeros))(x.detach().expand(2, rows, K2))
    assert float((y2.double() - want).norm() / want.norm()) <= 1e-3
    assert float((yt[1].double() - (want - bias.double() - res.double())[0]).norm() / want.norm()) <= 1e-3
    assert quant_cuda.device_status() == 0


@pytest.mark.parametrize("fmt", ["seq", "v1"])
@pytest.mark.parametrize("rows", [4, 40])
def test_skip_path_is_added_as_torch_adds_it(fmt, rows):
    """A skip path of another shape than the product's broadcasts (a row, more leading dimensions), one that is not
    contiguous or off a 16-byte boundary is added all the same, and a forward-mode tangent that it carries is kept."""
    mod, w, bias = build(fmt, 128 if fmt == "seq" else K)
    gen = torch.Generator().manual_seed(rows)
    x, full = torch.randn(rows, K, generator=gen).half().to(DEV), torch.randn(rows, N, generator=gen).half().to(DEV)
    off = torch.zeros(rows * N + 1, dtype=torch.float16, device=DEV)[1:].view(rows, N)
    off.copy_(full)
    with torch.no_grad():
        plain = mod(x)
        for res in (full[:1], full[0], full[None], full.t().contiguous().t(), off, full.float()):
            mod.offer_residual(res)
            y = mod(x)
            want = plain + res.half()
            assert y.shape == want.shape and torch.equal(y, want)
        with torch.autograd.forward_ad.dual_level():
            mod.offer_residual(torch.autograd.forward_ad.make_dual(full, full))
            assert torch.equal(torch.autograd.forward_ad.unpack_dual(mod(x)).tangent, full)
    assert quant_cuda.device_status() == 0


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_first_format_on_the_pair_kernel(variant):
    """Above 1024 rows, and wherever the pair kernel is asked for, a first-format layer runs on it with neither packed zero
    points nor g_idx: same product, scales of either sign and above 2 among them."""
    rows, K2, N2 = 1100, 1280, 768
    gen = torch.Generator().manual_seed(variant)
    qweight = torch.randint(-2 ** 31, 2 ** 31 - 1, (K2 // 8, N2), generator=gen).to(torch.int32).to(DEV)
    scales = (torch.rand(N2, 1, generator=gen) * 0.018 + 0.002).half()
    scales[::7] = -3.25 * scales[::7]
    scales[3::31] = 2.5
    zeros = (scales.float() * torch.randint(1, 16, (N2, 1), generator=gen)).half().to(DEV)
    scales, bias = scales.to(DEV), torch.randn(N2, generator=gen).half().to(DEV)
    x, res = torch.randn(rows, K2, generator=gen).half().to(DEV), torch.randn(rows, N2, generator=gen).half().to(DEV)
    w = torch.empty((K2, N2), dtype=torch.float16, device=DEV)
    quant_cuda.vecquant4recons_v1(qweight, w, scales.reshape(-1), zeros.reshape(-1))
    want = x.double() @ w.double() + bias.double() + res.double()
    quant_cuda.gemm_set_variant(variant)
    try:
        with torch.no_grad():
            y = quant_cuda.gemm_v1_new(x, qweight, scales, zeros, bias, res)
    finally:
        quant_cuda.gemm_set_variant(0)
    assert float((y.double() - want).norm() / want.norm()) <= 1e-3          # fp32 sums rounded to fp16 twice: 2 * 2^-11
    assert quant_cuda.device_status() == 0
