"""The work whose speed matters to a user of this framework, as a list of cases.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` builds what a
program holds before the call (model parts, weights, activations, a captured step), ``run(state)`` is one pass through
the public entry points, ``work(case)`` the bytes and operations the pass cannot do without and ``tolerance(case)``
how far two correct implementations may be apart.

Four kinds of work, all over GPTQ layers of LLaMA decoder blocks (hidden size, width of k and v, MLP width):

``linears``  inference through the quantised projections of ``layers`` decoder blocks: q, k, v, o, gate, up, down as
             ``Autograd4bitQuantLinear`` modules, or (``fused``) one qkv projection and ``QuantLlamaMLP``.  ``rows``
             tokens at once: 1 = generation, 2..16 = batched generation, more = a prompt.  ``part`` "attn" takes one
             square projection alone, the smallest call there is.  ``graph``: the program captured its step once as a
             CUDA graph, as servers do for generation; otherwise the modules are called one after the other.
``model``    a prompt through a whole patched LLaMA (fused attention and MLP, fused norms and rotary embedding).
``train``    forward and backward through the projections with grad enabled, LoRA factors on all seven (``lora`` > 0)
             or gradients for the input only (``lora`` 0, what a frozen projection does inside a finetune step).
``step``     a whole LoRA finetune step (``LoraFinetuner``): forward, backward under checkpointing, AdamW.

Layer formats: GPTQ v2 with groups of ``groupsize`` rows (-1: one group), sequential or permuted (``act_order``), and
the older v1 format (one scale and one float zero per column).
"""
from __future__ import annotations

import math

import torch
import torch.nn as nn

from alpaca_lora_4bit_b200 import fused_ops, matmul_utils_4bit
from alpaca_lora_4bit_b200 import finetune_step as ft
from alpaca_lora_4bit_b200.autograd_4bit import Autograd4bitQuantLinear
from alpaca_lora_4bit_b200.model_attn_mlp_patch import QuantLlamaMLP, fuse_quant_linears, make_fused_mlp, make_quant_attn
from alpaca_lora_4bit_b200.models import Linear4bitLt, adopt_packed_buffers

_LLAMA_7B = dict(hidden=4096, kv=4096, inter=11008)
_LLAMA_13B = dict(hidden=5120, kv=5120, inter=13824)
_LLAMA_70B = dict(hidden=8192, kv=1024, inter=28672)


def _linears(shape, rows, layers, groupsize=128, act_order=False, v1=False, fused=False, graph=False, part="block"):
    return dict(kind="linears", rows=rows, layers=layers, groupsize=groupsize, act_order=act_order, v1=v1, fused=fused,
                graph=graph, part=part, **shape)


def _model(shape, rows, layers):
    return dict(kind="model", rows=rows, layers=layers, **shape)


def _train(shape, rows, layers, lora, groupsize=128, act_order=False, bf16=False):
    return dict(kind="train", rows=rows, layers=layers, groupsize=groupsize, act_order=act_order, lora=lora, bf16=bf16, **shape)


def _step(shape, batch, seq, layers, lora, targets, act_order=False):
    return dict(kind="step", batch=batch, seq=seq, layers=layers, lora=lora, targets=targets, act_order=act_order, **shape)


def listed():
    return [
        # one projection of one token: the smallest call, all latency
        dict(_linears(_LLAMA_7B, 1, 1, part="attn"), name="one_projection_row"),
        # generation of one sequence, called module by module as transformers does
        dict(_linears(_LLAMA_7B, 1, 2, fused=True), name="token_7b_modules"),
        # the same from a captured step
        dict(_linears(_LLAMA_7B, 1, 4, graph=True), name="token_7b_graph"),
        # generation on an act-order checkpoint (the usual form of published 13B and larger GPTQ files)
        dict(_linears(_LLAMA_13B, 1, 2, act_order=True, graph=True), name="token_13b_act_order"),
        # batched generation: seven sequences at once
        dict(_linears(_LLAMA_13B, 7, 2, graph=True), name="tokens7_13b"),
        # a short prompt of 77 tokens
        dict(_linears(_LLAMA_7B, 77, 2), name="prompt77_7b"),
        # a prompt of ragged length on an act-order checkpoint
        dict(_linears(_LLAMA_13B, 333, 1, act_order=True, fused=True), name="prompt333_13b_act_order"),
        # a prompt on a checkpoint of the first format
        dict(_linears(_LLAMA_7B, 500, 1, groupsize=-1, v1=True), name="prompt500_7b_v1"),
        # a full context through a whole model
        dict(_model(_LLAMA_7B, 2048, 2), name="context2048_7b_model"),
        # several contexts at once through the largest layers, grouped-query attention: the largest product
        dict(_linears(_LLAMA_70B, 4096, 1), name="context4096_70b"),
        # finetuning with adapters on all projections of an act-order checkpoint, bf16 activations
        dict(_train(_LLAMA_13B, 2048, 1, 16, act_order=True, bf16=True), name="train2048_13b_act_order"),
        # the finetune step of the small configuration: 4 sequences of 256 tokens, adapters on q and v
        dict(_step(_LLAMA_7B, 4, 256, 3, 8, "q_proj,v_proj"), name="finetune_step_7b"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng):
    pick = rng.random()
    if pick < 0.5:
        return dict(rng.choice([_LLAMA_7B, _LLAMA_13B, _LLAMA_70B]))
    # other widths, and widths split over several GPUs: hidden a multiple of 256, the rest multiples of 128
    hidden = 256 * _log_int(rng, 8, 32)
    heads = hidden // 128
    kv = hidden if rng.random() < 0.5 else 128 * max(n for n in range(1, max(1, heads // 8) + 1) if heads % n == 0)
    return dict(hidden=hidden, kv=kv, inter=128 * int(round(hidden * rng.uniform(1.3, 3.5) / 128)))


def draw(rng):
    while True:
        shape = _draw_shape(rng)
        kind = rng.choices(["token", "tokens", "prompt", "context", "model", "train", "step"], [3, 3, 3, 2, 1, 3, 1])[0]
        groupsize = rng.choices([128, 64, 32, -1], [6, 1, 1, 1])[0]
        act_order = groupsize > 0 and rng.random() < 0.35
        v1 = groupsize < 0 and rng.random() < 0.5
        fused = rng.random() < 0.4
        if kind == "token":
            case = _linears(shape, 1, rng.randint(1, 3), groupsize, act_order, v1, fused, rng.random() < 0.5,
                            "attn" if rng.random() < 0.2 else "block")
        elif kind == "tokens":
            case = _linears(shape, rng.randint(2, 16), rng.randint(1, 2), groupsize, act_order, v1, fused, rng.random() < 0.5)
        elif kind == "prompt":
            case = _linears(shape, _log_int(rng, 17, 512), rng.randint(1, 2), groupsize, act_order, v1, fused)
        elif kind == "context":
            case = _linears(shape, _log_int(rng, 512, 4096), 1, groupsize, act_order, v1, fused)
        elif kind == "model":
            case = _model(shape, _log_int(rng, 64, 2048), rng.randint(1, 2))
        elif kind == "train":
            case = _train(shape, _log_int(rng, 128, 4096), 1, rng.choice([0, 8, 16, 32]), groupsize, act_order, rng.random() < 0.4)
        else:
            case = _step(shape, rng.randint(1, 4), 8 * rng.randint(16, 64), rng.randint(1, 3), rng.choice([8, 16]),
                         rng.choice(["q_proj,v_proj", "q_proj,k_proj,v_proj,o_proj,gate_proj,up_proj,down_proj"]), rng.random() < 0.35)
        largest = listed()[9]
        if work(case)["flops"] <= work(largest)["flops"]:
            return case


# ------------------------------------------------------------------------------------------------ shapes and work


def _projections(case):
    """(name, K, N) of the quantised projections of one decoder block."""
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    if case.get("part") == "attn":
        return [("o", h, h)]
    return [("q", h, h), ("k", h, kv), ("v", h, kv), ("o", h, h), ("gate", h, i), ("up", h, i), ("down", i, h)]


def _packed_bytes(case, K, N):
    if case.get("v1"):
        return K * N // 2 + 4 * N
    g = case.get("groupsize", 128)
    G = math.ceil(K / (g if g > 0 else K))
    return K * N // 2 + G * N // 2 + 2 * G * N + (4 * K if case.get("act_order") else 0)


def work(case):
    kind, layers = case["kind"], case["layers"]
    rows = case["batch"] * case["seq"] if kind == "step" else case["rows"]
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    proj = _projections(case)
    params = layers * sum(K * N for _, K, N in proj)
    weights = layers * sum(_packed_bytes(case, K, N) for _, K, N in proj)
    act_in = layers * 2 * rows * (3 * h + i if len(proj) > 1 else h)         # block input, attention output, MLP input, MLP middle
    act_out = layers * 2 * rows * sum(N for _, K, N in proj)
    flops = 2 * rows * params
    if kind == "linears":
        if case["fused"] and len(proj) > 1:                                  # the MLP's middle stays inside QuantLlamaMLP
            act_in, act_out = layers * 2 * rows * 3 * h, layers * 2 * rows * (h + 2 * kv + 2 * h)
        return {"bytes": weights + act_in + act_out, "flops": flops}
    if kind == "model":
        attn = layers * 2 * rows * rows * h                                  # causal: half of two products of rows x rows x h
        vocab = 2 * _VOCAB * h
        return {"bytes": weights + vocab + 4 * rows * h, "flops": flops + attn + vocab}
    if kind == "train":
        r = case["lora"]
        factors = layers * 4 * r * sum(K + N for _, K, N in proj)
        lora_flops = 3 * 2 * rows * r * layers * sum(K + N for _, K, N in proj)
        return {"bytes": 2 * weights + 2 * (act_in + act_out) + 2 * factors, "flops": 2 * flops + lora_flops}
    # step: forward and input gradients of the projections (nothing recomputed), attention forward and backward, lm_head both ways
    head = 2 * 2 * rows * _VOCAB * h
    attn = layers * 3.5 * 2 * rows * case["seq"] * h
    trained = layers * case["lora"] * sum(K + N for n, K, N in proj if n + "_proj" in case["targets"].split(","))
    return {"bytes": 2 * weights + 2 * _VOCAB * h * 2 + 4 * rows * _VOCAB + 28 * trained, "flops": 2 * flops + head + attn + 6 * rows * trained}


def tolerance(case):
    # about four times what these paths differ by from dense products in 32 bits of the weights dequantised to fp16
    if case["kind"] == "linears":                # fp16 results (5.5e-4: the fp16 rounding of the weights; 9.7e-4 after the SwiGLU product)
        return {"rel": 4e-3 if case["fused"] else 2.2e-3, "max": 0.02}
    if case["kind"] == "model":                  # a chain of fp16 layers: 3.4e-3, largest 0.05
        return {"rel": 1.4e-2, "max": 0.2}
    if case["kind"] == "train":                  # 5.2e-4 and 5e-3; sums of input gradients in bf16: 4.3e-3 and 0.04
        return {"rel": 1.7e-2, "max": 0.15} if case["bf16"] else {"rel": 2.2e-3, "max": 0.02}
    # losses, gradients and weights after a few optimiser steps: 1.0e-3, largest 0.07 (an AdamW step of a gradient near
    # zero may take either sign)
    return {"rel": 4e-3, "max": 0.28}


# ------------------------------------------------------------------------------------------------ building

_VOCAB = 32000


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _fill(mod, gen, act_order):
    gain = 1.0 / (6.3 * 0.011 * math.sqrt(mod.in_features))                  # unit gain, as trained layers roughly have
    if not mod.is_v1_model:
        return ft.fill_random_quant(mod, gen, act_order, scale_mul=gain)
    dev, K, N = gen.device, mod.in_features, mod.out_features
    mod.qweight = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // 8, N), generator=gen, device=dev, dtype=torch.int64).to(torch.int32)
    mod.scales = ((torch.rand((N, 1), generator=gen, device=dev) * 0.018 + 0.002) * gain).half()
    mod.zeros = (mod.scales.float() * torch.randint(1, 16, (N, 1), generator=gen, device=dev)).half()
    mod.bias = torch.zeros(N, dtype=torch.float16, device=dev)


def _make_linear(case, K, N, gen):
    with torch.device("meta"):
        mod = Autograd4bitQuantLinear(K, N, groupsize=case.get("groupsize", 128), is_v1_model=case.get("v1", False))
    mod.qweight = torch.empty((K // 8, N), dtype=torch.int32, device=gen.device)   # the device the contents are drawn on
    _fill(mod, gen, case["act_order"])
    return mod.requires_grad_(False).eval()


class _PlainMLP(nn.Module):
    def __init__(self, gate, up, down):
        super().__init__()
        self.gate_proj, self.up_proj, self.down_proj, self.act_fn = gate, up, down, nn.SiLU()


def _acts(gen, *shape, dtype=torch.float16):
    return torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float32).to(dtype)


def _prepare_linears(case, gen):
    mods, calls = [], []
    for _ in range(case["layers"]):
        lin = {n: _make_linear(case, K, N, gen) for n, K, N in _projections(case)}
        rows, h, i = case["rows"], case["hidden"], case["inter"]
        if case["part"] == "attn":
            calls.append((lin["o"], _acts(gen, rows, h)))
        elif case["fused"]:
            if case["act_order"]:                                            # projections of one input share their permutation
                for n in ("k", "v"):
                    lin[n].g_idx = lin["q"].g_idx
                lin["up"].g_idx = lin["gate"].g_idx
            qkv = fuse_quant_linears([lin["q"], lin["k"], lin["v"]], is_v1_model=case["v1"])
            mlp = QuantLlamaMLP(_PlainMLP(lin["gate"], lin["up"], lin["down"]), is_v1_model=case["v1"])
            calls += [(qkv, _acts(gen, rows, h)), (lin["o"], _acts(gen, rows, h)), (mlp, _acts(gen, rows, h))]
        else:
            x, a, m, d = _acts(gen, rows, h), _acts(gen, rows, h), _acts(gen, rows, h), _acts(gen, rows, i)
            calls += [(lin["q"], x), (lin["k"], x), (lin["v"], x), (lin["o"], a), (lin["gate"], m), (lin["up"], m), (lin["down"], d)]
    state = {"case": case, "calls": calls}
    if case["graph"]:
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _run_linears(state)
            _run_linears(state)
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            state["outputs"] = _run_linears(state)
        state["graph"] = graph
    return state


def _run_linears(state):
    # act-order checkpoints are served with the module-level switch on, as the reference's loader sets it
    matmul_utils_4bit.act_order = state["case"]["act_order"]
    try:
        with torch.no_grad():
            return [mod(x) for mod, x in state["calls"]]
    finally:
        matmul_utils_4bit.act_order = False


def _llama_shape(case):
    return ft.LlamaShape(hidden_size=case["hidden"], intermediate_size=case["inter"], num_hidden_layers=case["layers"],
                         num_attention_heads=case["hidden"] // 128, num_key_value_heads=case["kv"] // 128, vocab_size=_VOCAB,
                         max_position_embeddings=4096)


def _prepare_model(case, gen, seed):
    model = ft.build_quant_llama(_llama_shape(case), gen.device, seed=seed)
    cache = matmul_utils_4bit.cache_buffer
    make_quant_attn(model)
    matmul_utils_4bit.cache_buffer = cache
    make_fused_mlp(model)
    fused_ops.patch_llama(model)
    model.eval().requires_grad_(False)
    ids = torch.randint(0, _VOCAB, (1, case["rows"]), generator=gen, device=gen.device)
    return {"case": case, "model": model, "ids": ids}


def _run_model(state):
    # what generation does with a prompt: all hidden states, logits of the last position
    model = state["model"]
    with torch.no_grad():
        hidden = model.model(input_ids=state["ids"], use_cache=False).last_hidden_state
        return {"hidden": hidden, "logits": model.lm_head(hidden[:, -1])}


def _prepare_train(case, gen):
    dtype = torch.bfloat16 if case["bf16"] else torch.float16
    rows, h, i, r = case["rows"], case["hidden"], case["inter"], case["lora"]
    groups = []
    for _ in range(case["layers"]):
        lin = {}
        for n, K, N in _projections(case):
            mod = _make_linear(case, K, N, gen)
            if r:
                lora = Linear4bitLt("default", K, N, groupsize=case["groupsize"], r=r, lora_alpha=2 * r, lora_dropout=0.0)
                adopt_packed_buffers(lora, mod)
                a, b = lora.lora_A["default"].weight, lora.lora_B["default"].weight
                a.data = torch.randn((r, K), generator=gen, device=gen.device) * 0.02
                b.data = torch.randn((N, r), generator=gen, device=gen.device) * 0.02
                mod = lora.train()
            lin[n] = mod
        for names, K in ((("q", "k", "v"), h), (("o",), h), (("gate", "up"), h), (("down",), i)):
            x = _acts(gen, rows, K, dtype=dtype).requires_grad_(True)
            groups.append((x, [(lin[n], _acts(gen, rows, lin[n].out_features)) for n in names]))
    return {"case": case, "groups": groups}


def _run_train(state):
    bf16 = state["case"]["bf16"]
    out = []
    with torch.autocast("cuda", dtype=torch.bfloat16 if bf16 else torch.float16):
        for x, mods in state["groups"]:
            ys = [mod(x) for mod, _ in mods]
            wanted = [x] + [p for mod, _ in mods for p in mod.parameters() if p.requires_grad]
            grads = torch.autograd.grad(ys, wanted, [dy.to(y.dtype) for y, (_, dy) in zip(ys, mods)])
            out.append([y.detach() for y in ys] + list(grads))
    return out


def _prepare_step(case, gen, seed):
    # hidden states of unit size and layers that add a little to them, as in trained models: random layers at full gain
    # amplify the rounding of one layer by orders of magnitude on the way back through the next
    model = ft.build_quant_llama(_llama_shape(case), gen.device, act_order=case["act_order"], seed=seed, gain=0.25)
    with torch.no_grad():
        model.get_input_embeddings().weight.mul_(50.0)
    ft.add_lora(model, case["targets"].split(","), r=case["lora"], alpha=2 * case["lora"], seed=seed + 1)
    model.train()
    fused_ops.patch_llama(model, fuse_gate_up=True)
    ft.apply_gradient_checkpointing(model)
    ids = torch.randint(0, _VOCAB, (case["batch"], case["seq"]), generator=gen, device=gen.device)
    tuner = ft.LoraFinetuner(model, lr=3e-4)
    tuner.capture(ids)
    return {"case": case, "tuner": tuner, "ids": ids}


def _run_step(state):
    tuner = state["tuner"]
    loss = tuner.step(state["ids"])
    return {"loss": loss, "gradients": tuner.flat.buffer, "weights": tuner.opt.param}


# ------------------------------------------------------------------------------------------------ entry points


def prepare(case, seed):
    gen = torch.Generator(device=_device()).manual_seed(seed)
    if case["kind"] == "linears":
        return _prepare_linears(case, gen)
    if case["kind"] == "model":
        return _prepare_model(case, gen, seed)
    if case["kind"] == "train":
        return _prepare_train(case, gen)
    return _prepare_step(case, gen, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "linears":
        if "graph" in state:
            state["graph"].replay()
            return state["outputs"]
        return _run_linears(state)
    if kind == "model":
        return _run_model(state)
    if kind == "train":
        return _run_train(state)
    return _run_step(state)
