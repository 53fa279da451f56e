"""Workloads of the decoder's MoE path as a host program drives them through the package's public calls.

A case is one pass of one of these programs:

  layer   one `Context.layer_forward_normed` call: a decoder whose attention runs elsewhere calls each MoE layer by itself
  stack   one `Context.stack_forward` call over the eleven MoE layers
  host    one `Context.stack_forward_host` call: host buffers in, host buffers out, the copies included
  step    everything of a decoder pass that is not attention: layer 0's dense MLP, the eleven MoE layers call by call, the
          final norm and the LM head's argmax (over every row of a call of up to four tokens, which is a decode step of
          that many requests, and over the last row of a longer call, which is the prefill of a prompt)

All cases have the model's shapes.  What varies is the number of tokens (one for a decode step, tens for batched decode
or a short prompt, hundreds for a page, thousands for several pages at once), the storage type of the weights and how
evenly the router spreads the tokens over the experts.
"""
from __future__ import annotations

import importlib.util
import math
import os
import random
import sys
import types

import numpy as np
import torch

H, E, K, F, S = 1280, 64, 6, 896, 1792          # one MoE layer: hidden, experts, top-k, expert width, shared width
DENSE, VOCAB, LAYERS = 6848, 129280, 11         # layer 0's dense MLP, the vocabulary, the number of MoE layers
GROUP, STD, EPS = 64, 0.02, 1e-6
QTYPES = {"f16": 1, "q8_0": 3, "q4_0": 4}


def _package():
    """The package; its folder's name is no identifier."""
    name = "unlimitedocr_c_b200"
    if name not in sys.modules:
        root = os.path.join(os.getcwd(), "unlimitedocr.c_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"), submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # the smallest call: one token through one layer, the call between two attention steps of a greedy decode
        {"name": "layer_1_q4", "kind": "layer", "qtype": "q4_0", "tokens": 1, "routing": "even"},
        # the headline: one token through the eleven layers in one call
        {"name": "stack_1_q4", "kind": "stack", "qtype": "q4_0", "tokens": 1, "routing": "even"},
        # the same from host memory to host memory, as an engine without device buffers of its own calls it
        {"name": "host_1_q4", "kind": "host", "qtype": "q4_0", "tokens": 1, "routing": "even"},
        # a whole decode step of one request in the eight-bit profile
        {"name": "step_1_q8", "kind": "step", "qtype": "q8_0", "tokens": 1, "routing": "even"},
        # a few requests (or beams) decoded together from an unquantised model file
        {"name": "layer_3_f16", "kind": "layer", "qtype": "f16", "tokens": 3, "routing": "even"},
        # batched decode of eight requests whose tokens favour some experts
        {"name": "layer_8_q8", "kind": "layer", "qtype": "q8_0", "tokens": 8, "routing": "skewed"},
        # batched decode, an odd number of requests
        {"name": "layer_37_q4", "kind": "layer", "qtype": "q4_0", "tokens": 37, "routing": "skewed"},
        # a short prompt, or a batch just above the batched decode range
        {"name": "layer_77_q8", "kind": "layer", "qtype": "q8_0", "tokens": 77, "routing": "even"},
        # prefill of one page's vision and prompt tokens through everything but attention
        {"name": "step_907_q4", "kind": "step", "qtype": "q4_0", "tokens": 907, "routing": "zipf"},
        # several pages at once, popular and rare experts
        {"name": "layer_4096_q4", "kind": "layer", "qtype": "q4_0", "tokens": 4096, "routing": "zipf"},
        # the same from an unquantised model file, a ragged number of rows
        {"name": "layer_2049_f16", "kind": "layer", "qtype": "f16", "tokens": 2049, "routing": "zipf"},
        # the largest: eight requests of 2048 tokens in one call
        {"name": "layer_16384_q4", "kind": "layer", "qtype": "q4_0", "tokens": 16384, "routing": "even"},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["layer", "layer", "layer", "stack", "host", "step"])
    qtype = rng.choice(["q4_0", "q8_0", "f16"] if kind == "layer" else ["q4_0", "q8_0"])
    most = {"layer": 4096 if qtype == "f16" else 16384, "stack": 640, "host": 480, "step": 640}[kind]
    n = min(most, max(1, round(math.exp(rng.uniform(0.0, math.log(most))))))
    case = {"kind": kind, "qtype": qtype, "tokens": n, "routing": rng.choice(["even", "skewed", "zipf"])}
    return case if all({**c, **case} != c for c in listed()) else draw(rng)


# ------------------------------------------------------------------------------------------------------------- inputs

def _quantise(w: torch.Tensor, qtype: str):
    """(packed bytes, fp16 scales or None) of a [rows, cols] f32 matrix, as a model file stores them (host arrays)."""
    if qtype == "f16":
        return w.half().view(torch.uint8).reshape(-1).cpu().numpy(), None
    g = w.reshape(-1, GROUP)
    if qtype == "q8_0":
        scale = (g.abs().amax(1, keepdim=True) / 127.0).half()
        q = torch.round(g / scale.float()).clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    else:
        high, low = g.amax(1, keepdim=True), g.amin(1, keepdim=True)
        scale = (torch.where(high > -low, high, low) / -8.0).half()       # the largest value by magnitude becomes level -8
        q = torch.round(g / scale.float()).clamp_(-8, 7).add_(8.0).to(torch.uint8)
        q = q[:, : GROUP // 2] | (q[:, GROUP // 2:] << 4)
    return q.reshape(-1).cpu().numpy(), scale.reshape(-1).view(torch.int16).cpu().numpy().view(np.uint16)


def _normal(gen, rows: int, cols: int) -> torch.Tensor:
    return torch.randn((rows, cols), generator=gen, device="cuda", dtype=torch.float32).mul_(STD)


def _matrix(gen, rows: int, cols: int, qtype: str):
    w, s = _quantise(_normal(gen, rows, cols), qtype)
    return types.SimpleNamespace(qtype=QTYPES[qtype], rows=rows, cols=cols, qweight=w, qscale=s)


def _routing_bias(rng: np.random.Generator, routing: str):
    if routing == "even":
        return None
    if routing == "skewed":
        return rng.standard_normal(E).astype(np.float32)
    p = (rng.permutation(E) + 1.0) ** -1.1
    return np.log(p / p.sum()).astype(np.float32)


def _layer(gen, bias, qtype: str):
    # gate, up and down of an expert follow one another; down's [H][F] rows hold as many groups as gate's [F][H]
    w, s = _quantise(_normal(gen, E * 3 * F, H), qtype)
    router = _normal(gen, E, H).half().view(torch.int16).cpu().numpy().view(np.uint16)
    return types.SimpleNamespace(H=H, E=E, K=K, F=F, S=S, scaling=1.0, router=router, logit_bias=bias, expert_qtype=QTYPES[qtype],
                                 expert_qweight=w, expert_qscale=s, shared_gate=_matrix(gen, S, H, qtype),
                                 shared_up=_matrix(gen, S, H, qtype), shared_down=_matrix(gen, H, S, qtype))


def prepare(case, seed):
    kind, qtype, n = case["kind"], case["qtype"], case["tokens"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    ctx = _package().Context()
    s = types.SimpleNamespace(ctx=ctx, kind=kind, n=n, layers=1 if kind == "layer" else LAYERS)
    for _ in range(s.layers):
        ctx.map_layer(_layer(gen, _routing_bias(rng, case["routing"]), qtype))
    ctx.allocate_runtime_arenas(n)
    if kind == "host":
        s.x = torch.randn((n, H), generator=gen, device="cuda").half().view(torch.int16).cpu().numpy().view(np.uint16)
        return s
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    s.x = torch.randn((n, H), generator=gen, device="cuda").half()
    s.norms = [torch.rand(H, generator=gen, device="cuda").add_(0.5).half() for _ in range(LAYERS + 2)]
    s.out = torch.zeros((n, H), dtype=torch.float16, device="cuda")
    if kind == "step":
        s.dense = ctx.map_dense_mlp(_matrix(gen, DENSE, H, qtype), _matrix(gen, DENSE, H, qtype), _matrix(gen, H, DENSE, qtype), n)
        ctx.map_lm_head(_matrix(gen, VOCAB, H, qtype))
        s.rows = [torch.zeros((n, H), dtype=torch.float16, device="cuda") for _ in range(2)]
        s.heads = n if n <= 4 else 1
        s.last = s.out[n - s.heads:]
        s.ids = torch.zeros(s.heads, dtype=torch.int32, device="cuda")
        s.scores = torch.zeros(s.heads, dtype=torch.float32, device="cuda")
    return s


def run(s):
    ctx, n = s.ctx, s.n
    if s.kind == "layer":
        ctx.layer_forward_normed(0, s.x, s.norms[0], EPS, n, s.out)
        return s.out
    if s.kind == "stack":
        ctx.stack_forward(0, s.layers, s.x, n, s.out)
        return s.out
    if s.kind == "host":
        return ctx.stack_forward_host(0, s.layers, s.x).view(np.float16)
    a, b = s.rows
    ctx.dense_mlp_forward_normed(s.dense, s.x, s.norms[0], EPS, n, a)
    for i in range(s.layers):
        ctx.layer_forward_normed(i, a, s.norms[1 + i], EPS, n, b)
        a, b = b, a
    ctx.rmsnorm(a, s.norms[1 + s.layers], EPS, n, H, s.out)
    ctx.lm_head_argmax(s.last, s.heads, s.ids, s.scores)
    return s.out, s.ids, s.scores


# --------------------------------------------------------------------------------------------------------------- work

def _matrix_bytes(rows: int, cols: int, qtype: str) -> float:
    return rows * cols * {"f16": 2.0, "q8_0": 1.0 + 2.0 / GROUP, "q4_0": 0.5 + 2.0 / GROUP}[qtype]


def _experts_used(n: int, routing: str) -> float:
    """How many experts a call of n tokens can be expected to select (router logits are N(0, STD^2 H) plus the bias)."""
    rng = np.random.default_rng(7)
    m, used = min(n, 2048), []
    for _ in range(8):
        bias = _routing_bias(rng, routing)
        logits = rng.standard_normal((m, E)) * STD * math.sqrt(H) + (0.0 if bias is None else bias)
        used.append(len(np.unique(np.argpartition(-logits, K - 1, axis=1)[:, :K])))
    return float(np.mean(used))


def work(case):
    kind, qtype, n = case["kind"], case["qtype"], case["tokens"]
    layers = 1 if kind == "layer" else LAYERS
    weights = E * H * 2 + _experts_used(n, case["routing"]) * 3 * _matrix_bytes(F, H, qtype) + 3 * _matrix_bytes(S, H, qtype)
    flops = 2.0 * n * (E * H + 3 * K * F * H + 3 * S * H)
    total, ops = layers * weights + 2 * n * H * 2, layers * flops
    if kind == "step":
        heads = n if n <= 4 else 1
        total += 3 * _matrix_bytes(DENSE, H, qtype) + _matrix_bytes(VOCAB, H, qtype)
        ops += 2.0 * n * 3 * DENSE * H + 2.0 * heads * VOCAB * H
    return {"bytes": total, "flops": ops}


def tolerance(case):
    # Activations, SwiGLU products and outputs are fp16 (2^-11 a rounding, a handful of roundings to a layer), sums are f32.
    # Eleven layers add their roundings up, and a near-tie of the router may fall the other way in one of them.
    return {"rel": 2e-3 if case["kind"] == "layer" else 6e-3}


# -------------------------------------------------------------------------------------------------------------- exact

def _values(w: np.ndarray, s, qtype: str) -> torch.Tensor:
    """The weights a model file's bytes stand for, flat, in 64 bits on the GPU."""
    raw = torch.from_numpy(w).cuda()
    if qtype == "f16":
        return raw.view(torch.float16).double()
    scale = torch.from_numpy(s.view(np.float16)).cuda().double().unsqueeze(1)
    if qtype == "q8_0":
        level = raw.view(torch.int8).double().reshape(-1, GROUP)
    else:
        raw = raw.reshape(-1, GROUP // 2)
        level = torch.cat([raw & 15, raw >> 4], 1).double() - 8.0
    return (level * scale).reshape(-1)


def _swiglu(x, gate, up, down):
    g = x @ gate.T
    return (g * torch.sigmoid(g) * (x @ up.T)) @ down.T


def _matrix_values(m, qtype: str) -> torch.Tensor:
    return _values(m.qweight, m.qscale, qtype).reshape(m.rows, m.cols)


def _moe(layer, qtype: str, x: torch.Tensor) -> torch.Tensor:
    router = torch.from_numpy(layer.router.view(np.float16)).cuda().double().reshape(E, H)
    logits = x @ router.T
    if layer.logit_bias is not None:
        logits += torch.from_numpy(layer.logit_bias).cuda().double()
    probs, ids = torch.softmax(logits, 1).topk(K, 1)
    out = _swiglu(x, _matrix_values(layer.shared_gate, qtype), _matrix_values(layer.shared_up, qtype),
                  _matrix_values(layer.shared_down, qtype))
    per_w, per_s = len(layer.expert_qweight) // E, 0 if layer.expert_qscale is None else len(layer.expert_qscale) // E
    for e in ids.unique().tolist():
        token, slot = (ids == e).nonzero(as_tuple=True)
        scale = None if per_s == 0 else layer.expert_qscale[e * per_s:(e + 1) * per_s]
        gate, up, down = _values(layer.expert_qweight[e * per_w:(e + 1) * per_w], scale, qtype).reshape(3, F * H)
        y = _swiglu(x[token], gate.reshape(F, H), up.reshape(F, H), down.reshape(H, F))
        out.index_add_(0, token, y * probs[token, slot].unsqueeze(1))
    return out


def exact(case, seed):
    """What `run` returns, in 64 bits throughout (no rounding of activations); no value for the arg-max ids."""
    kind, qtype, n = case["kind"], case["qtype"], case["tokens"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    layers = [_layer(gen, _routing_bias(rng, case["routing"]), qtype) for _ in range(1 if kind == "layer" else LAYERS)]
    x = torch.randn((n, H), generator=gen, device="cuda").half().double()
    if kind in ("stack", "host"):
        for layer in layers:
            x = x + _moe(layer, qtype, x)
        return x
    norms = [torch.rand(H, generator=gen, device="cuda").add_(0.5).half().double() for _ in range(LAYERS + 2)]

    def normed(v, i):
        return v / torch.sqrt(v.square().mean(1, keepdim=True) + EPS) * norms[i]

    if kind == "layer":
        return x + _moe(layers[0], qtype, normed(x, 0))
    dense = [_matrix_values(_matrix(gen, *shape, qtype), qtype) for shape in ((DENSE, H), (DENSE, H), (H, DENSE))]
    x = x + _swiglu(normed(x, 0), *dense)
    for i, layer in enumerate(layers):
        x = x + _moe(layer, qtype, normed(x, 1 + i))
    out = normed(x, 1 + LAYERS)
    heads = n if n <= 4 else 1
    scores = out[n - heads:] @ _matrix_values(_matrix(gen, VOCAB, H, qtype), qtype).T
    return out, None, scores.amax(1)
