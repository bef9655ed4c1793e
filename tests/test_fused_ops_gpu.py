"""The fused element-wise kernels (RMSNorm, SwiGLU, rotary embedding) against the stock transformers
computation they replace: operator by operator, forward and backward, and on a whole two-layer quantised
LLaMA (loss and LoRA gradients of the patched model against the unpatched one)."""
import copy

import pytest
import torch

from alpaca_lora_4bit_b200 import finetune_step as fs, fused_ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(a, b):
    a, b = a.double(), b.double()
    return float((a.detach() - b.detach()).norm() / b.detach().norm())


@pytest.mark.parametrize("rows,H", [(1024, 4096), (7, 8192), (33, 200)])
def test_rmsnorm_matches_stock(rows, H):
    g = torch.Generator(device=DEV).manual_seed(rows + H)
    x = (torch.randn((rows, H), generator=g, device=DEV) * 3).half().requires_grad_(True)
    w = (1 + 0.1 * torch.randn(H, generator=g, device=DEV)).half()
    dy = torch.randn((rows, H), generator=g, device=DEV).half()
    y = fused_ops.rms_norm(x, w, 1e-5)
    y.backward(dy)
    got_dx = x.grad.clone(); x.grad = None
    h = x.to(torch.float32)
    ref = w * (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5)).to(torch.float16)
    ref.backward(dy)
    assert rel(y, ref) <= 1e-3 and float((y.detach().float() - ref.detach().float()).abs().max()) <= 2e-2      # same two roundings; the sums differ in order
    assert rel(got_dx, x.grad) <= 2e-3
    # fp64 calculus as the arbiter: the fused backward is at least as close as the stock one
    x64 = x.detach().double().requires_grad_(True)
    y64 = w.double() * (x64 * torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-5))
    y64.backward(dy.double())
    assert rel(got_dx, x64.grad) <= 1.05 * rel(x.grad, x64.grad) + 1e-5


@pytest.mark.parametrize("rows,I,fused_input", [(1024, 11008, False), (5, 256, False), (300, 1024, True)])
def test_swiglu_matches_stock(rows, I, fused_input):
    g = torch.Generator(device=DEV).manual_seed(rows + I)
    if fused_input:                                              # the two halves of one gate_up output
        gu = (torch.randn((rows, 2 * I), generator=g, device=DEV) * 2).half().requires_grad_(True)
        gate, up = torch.split(gu, I, dim=-1)
    else:
        gate = (torch.randn((rows, I), generator=g, device=DEV) * 2).half().requires_grad_(True)
        up = torch.randn((rows, I), generator=g, device=DEV).half().requires_grad_(True)
    d = torch.randn((rows, I), generator=g, device=DEV).half()
    out = fused_ops.swiglu(gate, up)
    ref = torch.nn.functional.silu(gate) * up
    assert rel(out, ref) <= 1e-3
    leaves = [gu] if fused_input else [gate, up]
    got = torch.autograd.grad(out, leaves, d)
    want = torch.autograd.grad(ref, leaves, d)
    for a, b in zip(got, want):
        assert rel(a, b) <= 3e-3


@pytest.mark.parametrize("B,T,H,KV,D,TB", [(4, 256, 32, 32, 128, 1), (1, 77, 8, 2, 64, 1), (3, 40, 4, 4, 32, 3)])
def test_rope_matches_stock(B, T, H, KV, D, TB):
    """TB: batch of the cos / sin tables (1 = the tables of one sequence, broadcast over the batch, as the model passes them)."""
    g = torch.Generator(device=DEV).manual_seed(T + D)
    q = torch.randn((B, T, H * D), generator=g, device=DEV).half().requires_grad_(True)
    k = torch.randn((B, T, KV * D), generator=g, device=DEV).half().requires_grad_(True)
    ang = torch.rand((TB, T, D // 2), generator=g, device=DEV) * 6.28
    cos, sin = torch.cat([ang.cos(), ang.cos()], -1).half(), torch.cat([ang.sin(), ang.sin()], -1).half()
    qv, kv = q.view(B, T, H, D).transpose(1, 2), k.view(B, T, KV, D).transpose(1, 2)
    qe, ke = fused_ops.apply_rotary_pos_emb(qv, kv, cos, sin)
    c, s = cos.unsqueeze(1), sin.unsqueeze(1)
    qr, kr = qv * c + fused_ops._rotate_half(qv) * s, kv * c + fused_ops._rotate_half(kv) * s
    assert qe.shape == qr.shape and rel(qe, qr) <= 1e-3 and rel(ke, kr) <= 1e-3
    dq, dk = torch.randn_like(qr), torch.randn_like(kr)
    got = torch.autograd.grad([qe, ke], [q, k], [dq, dk])
    want = torch.autograd.grad([qr, kr], [q, k], [dq, dk])
    assert rel(got[0], want[0]) <= 2e-3 and rel(got[1], want[1]) <= 2e-3


def test_patched_llama_step_matches_stock():
    shape = fs.LlamaShape(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=8,
                          num_key_value_heads=4, vocab_size=1000, max_position_embeddings=256)

    def build(patched):
        model = fs.build_quant_llama(shape, DEV, groupsize=128, seed=3)
        fs.add_lora(model, ["q_proj", "v_proj"], r=8, alpha=16, seed=4)
        if patched:
            fused_ops.patch_llama(model)
        fs.apply_gradient_checkpointing(model)
        model.train()
        return fs.LoraFinetuner(model, lr=0.0, loss_scale=64.0, dynamic_scale=False)

    ids = torch.randint(0, 1000, (2, 64), generator=torch.Generator().manual_seed(9)).to(DEV)
    from transformers.models.llama import modeling_llama as ml
    stock_rope = ml.apply_rotary_pos_emb
    try:
        a = build(False)
        la = float(a.step(ids)); ga = a.flat.buffer.clone()
        b = build(True)
        lb = float(b.step(ids)); gb = b.flat.buffer.clone()
    finally:
        ml.apply_rotary_pos_emb = stock_rope
    assert abs(la - lb) <= 2e-3 * abs(la)
    assert rel(gb, ga) <= 2e-2


def test_skip_path_adds_in_the_projection_epilogues():
    """patch_llama hands the two residual adds of every decoder layer to o_proj / down_proj
    (``q4_gemm_fwd_residual``): same logits and same LoRA gradients as the model with the stock layer forward,
    where the adds are torch kernels; the product itself (quant_cuda.gemm with a residual) equals product + add to the bit."""
    from alpaca_lora_4bit_b200 import quant_cuda, synth
    layer = synth.make_layer(1024, 768, 128, False, seed=3).to(DEV)
    x = synth.make_acts(300, 1024, seed=4).to(DEV)
    res = synth.make_acts(300, 768, seed=5).to(DEV)
    bias = (torch.randn(768, generator=torch.Generator().manual_seed(6)) * 0.1).half().to(DEV)
    for variant in (0, 1, 2, 3):
        quant_cuda.gemm_set_variant(variant)
        try:
            plain = torch.empty(300, 768, dtype=torch.float16, device=DEV)
            quant_cuda.gemm(x, layer.qweight, plain, layer.scales, layer.qzeros, layer.g_idx, bias=bias)
            fused = torch.empty_like(plain)
            quant_cuda.gemm(x, layer.qweight, fused, layer.scales, layer.qzeros, layer.g_idx, bias=bias, residual=res)
        finally:
            quant_cuda.gemm_set_variant(0)
        assert torch.equal(fused, plain + res), variant

    ids = torch.randint(0, 256, (2, 96), generator=torch.Generator().manual_seed(8)).to(DEV)
    shape = fs.LlamaShape(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=8,
                          num_key_value_heads=4, vocab_size=256, max_position_embeddings=256)

    def run(patch_layers):
        model = fs.build_quant_llama(shape, DEV, groupsize=128, seed=2)
        fs.add_lora(model, ["q_proj", "v_proj", "o_proj", "down_proj"], r=8, alpha=16, seed=3)
        if patch_layers:
            fused_ops.patch_llama(model)
            assert "forward" in model.model.layers[0].__dict__
        fs.apply_gradient_checkpointing(model)
        model.train()
        ft = fs.LoraFinetuner(model, lr=0.0, loss_scale=64.0, dynamic_scale=False)
        loss = float(ft.step(ids))
        torch.cuda.synchronize()
        for layer_ in model.model.layers:                       # nothing is left behind on the projections
            assert "_q4_residual" not in layer_.self_attn.o_proj.__dict__ and "_q4_residual" not in layer_.mlp.down_proj.__dict__
        return loss, ft.flat.buffer.clone()

    stock_rope = __import__("transformers.models.llama.modeling_llama", fromlist=["x"]).apply_rotary_pos_emb
    try:
        loss_p, g_p = run(True)
    finally:
        __import__("transformers.models.llama.modeling_llama", fromlist=["x"]).apply_rotary_pos_emb = stock_rope
    loss_s, g_s = run(False)
    assert abs(loss_p - loss_s) <= 2e-3 * abs(loss_s)
    assert float((g_p - g_s).norm() / g_s.norm()) <= 2e-2


def test_fused_gate_up_trains_like_two_layers():
    """patch_llama(fuse_gate_up=True) replaces the MLPs (no adapter on gate / up) by the fused-gate/up module: same
    loss and same LoRA gradients as the model with two layers, through checkpointing and the whole finetune step;
    an MLP with an adapter on gate_proj is left alone."""
    from alpaca_lora_4bit_b200 import model_attn_mlp_patch as patch
    ids = torch.randint(0, 256, (2, 96), generator=torch.Generator().manual_seed(8)).to(DEV)
    shape = fs.LlamaShape(hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=8,
                          num_key_value_heads=4, vocab_size=256, max_position_embeddings=256)

    def run(fuse, targets):
        model = fs.build_quant_llama(shape, DEV, groupsize=128, seed=2)
        fs.add_lora(model, targets, r=8, alpha=16, seed=3)
        fused_ops.patch_llama(model, fuse_gate_up=fuse)
        n_fused = sum(isinstance(m, patch.QuantLlamaMLP) for m in model.modules())
        fs.apply_gradient_checkpointing(model)
        model.train()
        ft = fs.LoraFinetuner(model, lr=0.0, loss_scale=64.0, dynamic_scale=False)
        loss = float(ft.step(ids))
        torch.cuda.synchronize()
        return loss, ft.flat.buffer.clone(), n_fused

    stock_rope = __import__("transformers.models.llama.modeling_llama", fromlist=["x"]).apply_rotary_pos_emb
    try:
        loss_f, g_f, n_f = run(True, ["q_proj", "v_proj", "down_proj"])
        loss_s, g_s, n_s = run(False, ["q_proj", "v_proj", "down_proj"])
        _, _, n_adapter = run(True, ["q_proj", "gate_proj"])
    finally:
        __import__("transformers.models.llama.modeling_llama", fromlist=["x"]).apply_rotary_pos_emb = stock_rope
    assert n_f == 2 and n_s == 0 and n_adapter == 0
    assert abs(loss_f - loss_s) <= 2e-3 * abs(loss_s)
    assert float((g_f - g_s).norm() / g_s.norm()) <= 2e-2


@pytest.mark.parametrize("rows,I", [(300, 1024), (1024, 11008), (5, 8)])
def test_swiglu_on_a_fused_gate_up_tensor(rows, I):
    """swiglu_fused takes [gate | up] as one tensor and returns one gradient tensor for it: same values as the
    two-tensor form (and as the stock expression), no concatenation in the backward."""
    g = torch.Generator(device=DEV).manual_seed(rows + I)
    gu = (torch.randn((2, rows, 2 * I), generator=g, device=DEV) * 2).half().requires_grad_(True)
    d = torch.randn((2, rows, I), generator=g, device=DEV).half()
    out = fused_ops.swiglu_fused(gu)
    gate, up = torch.split(gu, I, dim=-1)
    assert torch.equal(out, fused_ops.swiglu(gate, up))
    ref = torch.nn.functional.silu(gate) * up
    assert rel(out, ref) <= 1e-3
    (got,) = torch.autograd.grad(out, [gu], d)
    (two,) = torch.autograd.grad(fused_ops.swiglu(gate, up), [gu], d)
    (want,) = torch.autograd.grad(ref, [gu], d)
    assert torch.equal(got, two) and rel(got, want) <= 3e-3


def test_swiglu_fused_is_no_opaque_call_where_torch_watches():
    """The no-gradient product is one native call only where nobody watches.  A tracer, which sees the sizes as tensors, is
    refused by the autograd function's library call, and forward mode as it is refused by every function without a jvp:
    an error, and not a trace that replays uninitialised memory or a tangent that is dropped."""
    gen = torch.Generator(device=DEV).manual_seed(2)
    a, b = (torch.randn(5, 256, generator=gen, device=DEV).half() for _ in range(2))
    for grad in (True, False):
        with torch.set_grad_enabled(grad):
            with pytest.raises(Exception):
                torch.jit.trace(fused_ops.swiglu_fused, (a,), check_trace=False)
            with torch.autograd.forward_ad.dual_level():
                with pytest.raises(Exception, match="jvp"):
                    fused_ops.swiglu_fused(torch.autograd.forward_ad.make_dual(a, b))
            assert torch.equal(fused_ops.swiglu_fused(a), fused_ops._SwiGLUFused.apply(a))


def _stock_loss(logits, labels, vocab_size, num_items_in_batch=None, ignore_index=-100, shift_labels=None, **kwargs):
    if shift_labels is None:
        shift_labels = torch.nn.functional.pad(labels, (0, 1), value=ignore_index)[..., 1:]
    return torch.nn.functional.cross_entropy(logits.float().reshape(-1, vocab_size), shift_labels.reshape(-1), ignore_index=ignore_index)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T,V,shifted", [(1, 1, 8, True), (2, 5, 32000, False), (3, 7, 4104, False), (1, 33, 128256, True), (4, 64, 4096, False)])
def test_causal_loss_matches_stock(B, T, V, shifted, dtype):
    """The mean cross entropy in fp32 and its gradient rounded once to the logits' type: sums of up to V exponentials in
    another order (V * 2^-24 at the very most, as for the framework's own), and the one rounding."""
    gen = torch.Generator(device=DEV).manual_seed(V + T)
    logits = (torch.randn((B, T, V), generator=gen, device=DEV) * 4).to(dtype).requires_grad_(True)
    labels = torch.randint(0, V, (B, T), generator=gen, device=DEV)
    if T > 2:
        labels[0, 2] = -100
    kw = dict(shift_labels=labels) if shifted else {}
    fused = fused_ops.causal_lm_loss(lambda *a, **k: (_ for _ in ()).throw(AssertionError("the stock loss ran")))
    got = fused(logits, labels, V, **kw)
    assert got.dtype == torch.float32 and got.dim() == 0
    (got * 1024).backward()
    dgot, logits.grad = logits.grad, None
    want = _stock_loss(logits, labels, V, **kw)
    (want * 1024).backward()
    if not shifted and T == 1:
        return
    assert abs(float(got.detach()) - float(want.detach())) <= 1e-6 * abs(float(want.detach())) + 1e-6
    l64 = logits.detach().double().requires_grad_(True)
    loss64 = torch.nn.functional.cross_entropy(l64.reshape(-1, V), (labels if shifted else torch.nn.functional.pad(labels, (0, 1), value=-100)[..., 1:]).reshape(-1))
    (loss64 * 1024).backward()
    assert rel(dgot, l64.grad) <= rel(logits.grad, l64.grad) * 1.02 + 1e-6
    assert float((dgot.float() - logits.grad.float()).abs().max()) <= 2 ** (-10 if dtype == torch.float16 else -7) * float(logits.grad.float().abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("offset", [0.0, 300.0, 1000.0, -20000.0])
def test_causal_loss_of_confident_rows_and_of_logits_with_an_offset(offset, dtype):
    """Against 64 bits on the same 16-bit logits.  fp32: log s of a sum s = 1 + eps carries a few 2^-24, absolute, so that
    softmax - 1 does too, however small it is; an exponent d (the log probability) two roundings, 2^-24 |d| each, which are
    relative errors of its exponential; the gradient is then rounded once to 16 bits.  (With the exponent formed as
    x log2(e) - m log2(e) the errors grew with the logits.)"""
    B, V = 16, 32000
    gen = torch.Generator(device=DEV).manual_seed(int(abs(offset)) + 1)
    x = torch.randn((B, V), generator=gen, device=DEV) * 2
    labels = torch.randint(0, V, (B,), generator=gen, device=DEV)
    x[torch.arange(B, device=DEV), labels] = 14 + 8 * torch.rand(B, generator=gen, device=DEV)      # probability 0.9 .. 0.9999
    logits = (x + offset).to(dtype).requires_grad_(True)
    fused = fused_ops.causal_lm_loss(lambda *a, **k: (_ for _ in ()).throw(AssertionError("the stock loss ran")))
    loss = fused(logits, None, V, shift_labels=labels)
    scale = 1024.0 * B
    (loss * scale).backward()
    l64 = logits.detach().double().requires_grad_(True)
    loss64 = torch.nn.functional.cross_entropy(l64, labels)
    (loss64 * scale).backward()
    assert abs(float(loss.detach()) - float(loss64.detach())) <= 8 * 2 ** -24 * (1 + float(loss64.detach()))
    got, want = logits.grad.double(), l64.grad
    hot, d = torch.nn.functional.one_hot(labels, V), torch.log_softmax(l64.detach(), 1).abs()
    tol = 2 ** (-11 if dtype == torch.float16 else -8) * want.abs() + 2 ** -24 * ((8 + 2 * d) * want.abs() + 8 * (scale / B) * hot)
    if dtype == torch.float16:
        tol = tol + 2 ** -25                             # half the smallest subnormal
    assert bool(((got - want).abs() <= tol * 1.001).all()), float(((got - want).abs() / tol).max())


@pytest.mark.parametrize("shifted", [False, True])
def test_causal_loss_keeps_what_its_backward_reads(shifted):
    """Logits and labels are the program's own: written to before the backward (as a sampler or the next batch does), they
    leave the gradient alone, once and again, as with the stock loss.  (The backward read them, and raised.)"""
    V = 512
    gen = torch.Generator(device=DEV).manual_seed(5)
    leaf = torch.randn((2, 9, V), generator=gen, device=DEV).half().requires_grad_(True)
    labels = torch.randint(0, V, (2, 9), generator=gen, device=DEV)
    labels[1, 4] = -100
    kw = lambda l: dict(labels=None, shift_labels=l) if shifted else dict(labels=l)
    (want,) = torch.autograd.grad(_stock_loss(leaf, vocab_size=V, **kw(labels)), leaf)
    fused = fused_ops.causal_lm_loss(lambda *a, **k: (_ for _ in ()).throw(AssertionError("the stock loss ran")))
    logits = leaf * 1
    given = labels.clone()
    loss = fused(logits, vocab_size=V, **kw(given))
    with torch.no_grad():
        logits.fill_(3.0)
        given.fill_(1)
    for last in (False, True):
        (got,) = torch.autograd.grad(loss, leaf, retain_graph=not last)
        assert rel(got, want) <= 2 ** -10
    with torch.no_grad():
        assert not fused(leaf, vocab_size=V, **kw(labels)).requires_grad


def test_causal_loss_has_a_second_derivative():
    """As the stock loss has, through the copy of the logits and through the gradient of the loss (it was refused)."""
    V = 64
    gen = torch.Generator(device=DEV).manual_seed(6)
    leaf = torch.randn((1, 5, V), generator=gen, device=DEV).half().requires_grad_(True)
    labels = torch.randint(0, V, (1, 5), generator=gen, device=DEV)
    labels[0, 2] = -100
    v = torch.randn(leaf.shape, generator=gen, device=DEV)
    out = []
    for f in (fused_ops.causal_lm_loss(_stock_loss), _stock_loss):
        scale = torch.tensor(64.0, device=DEV, requires_grad=True)
        (g,) = torch.autograd.grad(f(leaf, labels, V) * scale, leaf, create_graph=True)
        out.append((g, *torch.autograd.grad((g.float() * v).sum() + 3 * f(leaf, labels, V) * scale, (leaf, scale))))
    for a, b in zip(*out):
        assert a.shape == b.shape and rel(a, b) <= 2 ** -9


def test_causal_loss_at_the_edges():
    """No row with a class, infinities and NaN among the logits: what the framework's loss gives; the loss may be written in
    place before its backward; other calls go to the stock loss."""
    V = 64
    fused = fused_ops.causal_lm_loss(_stock_loss)
    none = torch.full((1, 4), -100, device=DEV)
    x = torch.randn((1, 4, V), device=DEV).half().requires_grad_(True)
    assert torch.isnan(fused(x, none, V))
    for special in (float("inf"), float("-inf"), float("nan")):
        for where in (3, slice(None)):
            y = torch.randn((1, 4, V), device=DEV).half()
            y[0, 1, where] = special
            labels = torch.tensor([[1, 2, 3, 4]], device=DEV)
            a, b = fused(y, labels, V), _stock_loss(y, labels, V)
            assert torch.allclose(a, b, rtol=0, atol=1e-5, equal_nan=True), (special, where, a, b)
    labels = torch.randint(0, V, (1, 4), device=DEV)
    loss = fused(x, labels, V)
    loss /= 2
    loss.backward()
    ref = x.detach().clone().requires_grad_(True)
    (_stock_loss(ref, labels, V) / 2).backward()
    assert rel(x.grad, ref.grad) <= 1e-3
    seen = []
    spy = fused_ops.causal_lm_loss(lambda *a, **k: seen.append(1) or _stock_loss(*a, **k))
    for args, kw in (((x.float(), labels, V), {}), ((x, labels, V), dict(num_items_in_batch=torch.tensor(4, device=DEV))),
                     ((x.transpose(0, 1).contiguous().transpose(0, 1), labels, V), dict(label_smoothing=0.0)), ((x.cpu(), labels.cpu(), V), {})):
        spy(*args, **kw)
    assert len(seen) == 4
