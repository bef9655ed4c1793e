"""What the host side of the native products checks before anything is launched; no GPU: operands are stand-ins with the
attributes of tensors, the native module is a stub."""
import os
import warnings

import pytest
import torch

from alpaca_lora_4bit_b200 import _lib, autograd_4bit as a4, matmul_utils_4bit as mm4b, quant_cuda, synth
from tests import fake_backend

K, N, G = 512, 256, 4


class Operand:
    """A tensor's attributes, as far as the host code looks."""

    def __init__(self, shape, dtype, device="cuda:0", contiguous=True):
        self.shape, self.dtype, self.device, self._contiguous = torch.Size(shape), dtype, torch.device(device), contiguous
        self.is_cuda = self.device.type == "cuda"
        self._version = 0

    def dim(self):
        return len(self.shape)

    def numel(self):
        return self.shape.numel()

    def is_contiguous(self):
        return self._contiguous

    def data_ptr(self):
        return 4096


class NativeStub:
    def __init__(self):
        self.calls = []

    def gemm(self, *args):
        self.calls.append(args)
        return None


@pytest.fixture
def native(monkeypatch):
    stub = NativeStub()
    monkeypatch.setattr(quant_cuda, "_current_device", lambda: 0)
    monkeypatch.setattr(quant_cuda, "_raw_stream", lambda idx: 0)
    monkeypatch.setattr(quant_cuda, "groups_are_sequential", lambda g_idx, groups: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(_lib, "_gemm_workspaces", {(0, 0): Operand((1 << 30,), torch.uint8)})
    monkeypatch.setattr(_lib, "_torch_call", stub)
    monkeypatch.setattr(quant_cuda, "_zero_term_tables", {})
    return stub


def operands(**kw):
    o = dict(x=Operand((32, K), torch.float16), qweight=Operand((K // 8, N), torch.int32), out=Operand((32, N), torch.float16),
             scales=Operand((G, N), torch.float16), zeros=Operand((G, N // 8), torch.int32), g_idx=Operand((K,), torch.int32))
    o.update(kw)
    return o


BAD = {
    "zeros on the CPU": dict(zeros=Operand((G, N // 8), torch.int32, "cpu")),
    "zeros on another GPU": dict(zeros=Operand((G, N // 8), torch.int32, "cuda:1")),
    "scales on another GPU": dict(scales=Operand((G, N), torch.float16, "cuda:1")),
    "scales too narrow": dict(scales=Operand((G, N // 2), torch.float16)),
    "zeros too narrow": dict(zeros=Operand((G, N // 16), torch.int32)),
    "zeros of fewer groups": dict(zeros=Operand((G - 1, N // 8), torch.int32)),
    "zeros not packed": dict(zeros=Operand((G, N // 8), torch.float16)),
    "scales not contiguous": dict(scales=Operand((G, N), torch.float16, contiguous=False)),
}


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("what", sorted(BAD))
def test_zero_term_table_is_not_made_from_operands_that_are_no_layer(native, monkeypatch, what, transpose):
    def launched(*args):
        raise AssertionError("the table kernel must not be launched")
    monkeypatch.setattr(_lib, "lib", lambda: type("Lib", (), {"q4_gemm_workspace_bytes": staticmethod(lambda *a: 0),
                                                              "q4_zero_term_table": staticmethod(launched)}))
    o = operands(**BAD[what])
    assert quant_cuda.gemm_new(o["x"], o["qweight"], o["out"], o["scales"], o["zeros"], o["g_idx"], transpose) is None
    assert quant_cuda._zero_terms(o["scales"], o["zeros"], G, N, 0) is None
    with pytest.raises(RuntimeError):                       # and the general path says what is wrong
        quant_cuda.gemm(o["x"], o["qweight"], o["out"], o["scales"], o["zeros"], o["g_idx"], transpose)
    assert quant_cuda._zero_term_tables == {}


def test_native_calls_stand_back_where_torch_watches():
    """Under a forward-mode level, a function transform or a tracer the opaque calls are not taken (the operators then go
    through their autograd functions, which those modes record, refuse or batch)."""
    x = torch.randn(3, 4)
    assert _lib.nobody_watches()
    seen = []

    def look(t):
        seen.append(_lib.nobody_watches())
        return t * 2

    with torch.autograd.forward_ad.dual_level():
        look(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))
    torch.func.vmap(look)(x)
    torch.func.grad(lambda t: look(t).sum())(x)
    torch.func.jvp(look, (x,), (x,))
    torch.jit.trace(look, (x,), check_trace=False)
    assert seen == [False] * 5
    assert _lib.nobody_watches()
    assert not _lib.opaque_call_ok(x)                       # and never for tensors that are not on a GPU


def small_module(**kw):
    layer = synth.make_layer(256, 64, 64, False, 1)
    mod = a4.Autograd4bitQuantLinear(256, 64, groupsize=64, **kw)
    mod.qweight, mod.qzeros, mod.scales, mod.g_idx = layer.qweight, layer.qzeros, layer.scales, layer.g_idx
    mod.bias = torch.randn(64, generator=torch.Generator().manual_seed(2)).half()
    return mod, synth.make_acts(3, 256, 5)


@pytest.mark.parametrize("how", ["parameter", "attribute", "parametrization"])
@pytest.mark.parametrize("name", ["scales", "qzeros", "g_idx", "qweight", "bias"])
def test_no_grad_forward_finds_operands_registered_as_something_else(name, how):
    with fake_backend.installed(), torch.no_grad():
        mod, x = small_module()
        want, value = mod(x), getattr(mod, name)
        if how == "parametrization":
            class Same(torch.nn.Module):
                def forward(self, t):
                    return t.clone()
            torch.nn.utils.parametrize.register_parametrization(mod, name, Same(), unsafe=True)
        else:
            delattr(mod, name)
            setattr(mod, name, torch.nn.Parameter(value, requires_grad=False) if how == "parameter" else value)
        assert name not in mod._buffers
        assert torch.equal(mod(x), want)


def test_no_grad_forward_calls_a_product_that_was_put_in_place(monkeypatch):
    mod, x = small_module()
    res = torch.randn(3, 64).half()
    seen = []

    def ones(x, *args):
        seen.append(args)
        return torch.ones(x.shape[:-1] + (64,), dtype=torch.float16)

    with torch.no_grad():
        for target, name in ((a4, "matmul4bit_with_backend"), (mm4b, "matmul4bit")):
            with monkeypatch.context() as m:
                m.setattr(target, name, ones)
                assert torch.equal(mod(x), 1 + mod.bias.expand(3, 64))
                mod.offer_residual(res)
                assert torch.equal(mod(x), (1 + mod.bias.expand(3, 64)) + res)
    assert len(seen) == 4 and all(a[0] is mod.qweight and a[2] is mod.qzeros for a in seen)


def test_skip_path_is_taken_through_the_method():
    class Sub(a4.Autograd4bitQuantLinear):
        def take_residual(self):
            super().take_residual()
            return None

    mod, x = small_module()
    with fake_backend.installed(), torch.no_grad():
        want = mod(x)
        mod.__class__ = Sub
        mod.offer_residual(torch.ones(3, 64).half())
        assert torch.equal(mod(x), want)


@pytest.fixture
def build_in(tmp_path, monkeypatch):
    """The build of the native module with its products in a folder of the test's own and the compiler a stub."""
    from alpaca_lora_4bit_b200 import build
    src = tmp_path / "q4torch.cpp"
    src.write_text("int one;")
    runs = []

    def compile_(cmd):
        runs.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("module")
    monkeypatch.setattr(build, "TORCH_SRC", str(src))
    monkeypatch.setattr(build, "TORCH_LIB", str(tmp_path / "_q4torch.so"))
    monkeypatch.setattr(build, "TORCH_KEY", str(tmp_path / "_q4torch.key"))
    monkeypatch.setattr(build.subprocess, "check_call", compile_)
    return build, src, runs


def test_native_module_is_built_again_when_its_sources_or_torch_change(build_in, monkeypatch):
    build, src, runs = build_in
    for _ in range(3):
        assert build.build_torch_call() == build.TORCH_LIB
    assert len(runs) == 1
    src.write_text("int two;")
    os.utime(src, (0, 0))                                   # an older file with other contents
    build.build_torch_call()
    build.build_torch_call()
    assert len(runs) == 2
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    build.build_torch_call()
    build.build_torch_call()
    assert len(runs) == 3
    os.remove(build.TORCH_LIB)
    build.build_torch_call()
    assert len(runs) == 4 and sorted(os.listdir(src.parent)) == ["_q4torch.key", "_q4torch.so", "q4torch.cpp"]


def test_without_the_native_module_the_ctypes_binding_serves(monkeypatch):
    from alpaca_lora_4bit_b200 import build

    def fails():
        raise RuntimeError("no C++ compiler")
    monkeypatch.setattr(build, "build_torch_call", fails)
    monkeypatch.setattr(_lib, "_torch_call", None)
    with pytest.warns(UserWarning, match="no C\\+\\+ compiler"):
        native = _lib.torch_call()
    with warnings.catch_warnings():
        warnings.simplefilter("error")                      # said once
        assert _lib.torch_call() is native
    assert native.gemm() is None and native.swiglu(1) is None and native.gemv(1, 2) is None and native.gemm_v1(1) is None


def test_order_of_groups_is_answered_per_group_count():
    """One g_idx asked with several group counts: each gets its own answer, also after it is written to."""
    g_idx = torch.zeros(256, dtype=torch.int32)
    for _ in range(2):
        assert quant_cuda.groups_are_sequential(g_idx, 1)
        assert not quant_cuda.groups_are_sequential(g_idx, 4)
        assert not quant_cuda.groups_are_sequential(g_idx, 3) and not quant_cuda.groups_are_sequential(g_idx, 0)
    g_idx.copy_(torch.arange(256) // 64)
    for _ in range(2):
        assert quant_cuda.groups_are_sequential(g_idx, 4)
        assert not quant_cuda.groups_are_sequential(g_idx, 1)


def test_zero_term_table_follows_the_scales_object(native, monkeypatch):
    """New scales at the address of freed ones, no writes counted on either: the table is made again."""
    made = []
    monkeypatch.setattr(_lib, "lib", lambda: type("Lib", (), {"q4_zero_term_table": staticmethod(lambda *a: made.append(a) or 0)}))
    monkeypatch.setattr(torch, "empty", lambda shape, dtype, device: Operand(shape, dtype, str(device)))
    zeros, first, second = operands()["zeros"], operands()["scales"], operands()["scales"]
    a = quant_cuda._zero_terms(first, zeros, G, N, 0)
    assert quant_cuda._zero_terms(first, zeros, G, N, 0) is a and len(made) == 1
    assert quant_cuda._zero_terms(second, zeros, G, N, 0) is not a and len(made) == 2


def test_decode_products_behind_a_cast_say_so(monkeypatch):
    """Scales (or first-format zeros) cast or copied for the call were written by the kernel just ahead: the product is
    told, so that it starts behind it."""
    flags = []
    monkeypatch.setattr(quant_cuda, "gemv", lambda x, qw, y, sc, zr, gi, gs, fl, bias=None: flags.append(bool(fl & _lib.GEMV_WRITTEN)) or y.zero_())
    layer = synth.make_layer(256, 64, 64, False, 1)
    x, y = synth.make_acts(3, 256, 5), torch.zeros(3, 64, dtype=torch.float16)
    for scales, said in ((layer.scales, False), (layer.scales.float(), True)):
        mm4b._matmul4bit_v2(x, layer.qweight, scales, layer.qzeros, layer.g_idx, 64)
        quant_cuda.vecquant4matmul_faster(x, layer.qweight, y, scales, layer.qzeros, layer.g_idx)
        quant_cuda.vecquant4matmul_old_faster(x, layer.qweight, y.float(), scales, layer.qzeros, 64)
        assert flags == [said] * 3
        flags.clear()
    one = layer.scales[:1].reshape(-1, 1).contiguous()
    for scales, zeros, said in ((one, one, False), (one.float(), one, True), (one, one.float(), True)):
        mm4b._matmul4bit_v1(x, layer.qweight, scales, zeros)
        quant_cuda.vecquant4matmul_v1_faster(x, layer.qweight, y, scales, zeros)
        assert flags == [said] * 2
        flags.clear()
