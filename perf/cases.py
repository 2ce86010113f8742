"""Performance cases of the framework: what a training or attribution run has it compute.

A case is a dict of plain values with a ``kind``:

* ``mlp_step``, ``gpt2_step`` -- one whole step of a user's loop: forward and backward over
  ``cat(train, val)`` with the engine's hooks attached, ``prepare_gradients``, ``aggregate_and_log``;
* ``dense``, ``norm``, ``embedding``, ``conv2d`` -- what the backward pass of one hooked layer costs: the
  hook bodies an engine registers, handed the (input, out-grad) pair that autograd hands them, between
  the two calls that open and close a backward pass.  Everything around it in a step is the model's own;
* ``gradproj``, ``gradproj_embedding`` -- the two hooks of a projected layer;
* ``similarity`` -- scores of one block of projected gradients against another.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges.
"""
from __future__ import annotations

import math

import torch
from torch import nn

from ghostsuite_b200.ghostEngines import GradDotProdEngine
from ghostsuite_b200.ghostEngines import autograd_grad_sample_dotprod as hooks
from ghostsuite_b200.ghostEngines import supported_layers_grad_samplers_dotprod as layers
from ghostsuite_b200.ghostEngines.gradProjection.autograd_gradproj import create_projection_hooks
from ghostsuite_b200.ghostEngines.gradProjection.projection_utils import (
    init_projection_matrix_gaussian, projection_similarity)
from ghostsuite_b200.workloads import GPT2Config, GPT2Like, make_mlp

_DT = {"bf16": torch.bfloat16, "fp32": torch.float32}
_SIZE = {"bf16": 2, "fp32": 4}


def listed():
    return [
        # the MLP configuration (512 -> 1024 -> 1024 -> 10, fp32, 64 + 16 samples): the smallest
        # step, all launches and host work
        {"name": "mlp_step_fp32", "kind": "mlp_step", "dtype": "fp32", "n_train": 64, "n_val": 16,
         "d_in": 512, "hidden": 1024, "d_out": 10},
        # a GPT-2-width decoder on a small share of the batch, as one rank of several sees it: every
        # layer type in one backward pass, bound by the host as much as by the GPU
        {"name": "gpt2_step_bf16", "kind": "gpt2_step", "dtype": "bf16", "n_train": 4, "n_val": 2, "T": 512,
         "layers": 4, "d": 768, "vocab": 50257},
        # GPT-2 small's MLP up-projection at the benchmark's batch: the layer shape a step meets most,
        # with its bias, per-sample path
        {"name": "conv1d_gpt2_fc_bf16", "kind": "dense", "layer": "conv1d", "bias": True, "dtype": "bf16",
         "n_train": 32, "n_val": 8, "T": 1024, "d_in": 768, "d_out": 3072},
        # the LM head of the same step: one layer with a third of its per-sample work
        {"name": "linear_gpt2_head_bf16", "kind": "dense", "layer": "linear", "bias": False, "dtype": "bf16",
         "n_train": 32, "n_val": 8, "T": 1024, "d_in": 768, "d_out": 50304},
        # the single-layer configuration at its shortest sequences: many samples of few tokens, Gram path
        {"name": "linear_wide_T128_bf16", "kind": "dense", "layer": "linear", "bias": False, "dtype": "bf16",
         "n_train": 256, "n_val": 32, "T": 128, "d_in": 4096, "d_out": 11008},
        # an fp32 model (the engines' default precision) with a token count and a width that fit no tile
        {"name": "linear_ragged_fp32", "kind": "dense", "layer": "linear", "bias": True, "dtype": "fp32",
         "n_train": 24, "n_val": 5, "T": 197, "d_in": 768, "d_out": 1000},
        # GPT-2 small's LayerNorm at the benchmark's batch
        {"name": "layernorm_gpt2_bf16", "kind": "norm", "rms": False, "dtype": "bf16", "n_train": 32, "n_val": 8,
         "T": 1024, "d": 768},
        # the token table of a language model: text has a few ids that fill a good part of every
        # sequence and a long tail
        {"name": "embedding_text_bf16", "kind": "embedding", "ids": "text", "dtype": "bf16", "n_train": 32,
         "n_val": 8, "T": 1024, "d": 768, "vocab": 50304},
        # a 3x3 convolution of a small image model, fp32
        {"name": "conv2d_3x3_fp32", "kind": "conv2d", "dtype": "fp32", "bias": True, "n_train": 64, "n_val": 16,
         "side": 16, "c_in": 64, "c_out": 128, "k": 3, "stride": 1},
        # GradProj on the Llama-3-8B gate projection: the largest operands of the projected models
        {"name": "gradproj_llama_gate_bf16", "kind": "gradproj", "layer": "linear", "dtype": "bf16", "batch": 8,
         "T": 4096, "d_in": 4096, "d_out": 14336, "k_i": 64, "k_o": 64},
        # GradProj of the token table of the Pythia-410M configuration
        {"name": "gradproj_embedding_bf16", "kind": "gradproj_embedding", "ids": "uniform", "dtype": "bf16",
         "batch": 16, "T": 2048, "d": 1024, "vocab": 50304, "k_i": 32, "k_o": 32},
        # similarity of two blocks of Pythia-410M projections (96 layers x 32 x 32)
        {"name": "similarity_64x64_fp32", "kind": "similarity", "dtype": "fp32", "n1": 64, "n2": 64, "dim": 98304},
    ]


# ------------------------------------------------------------------------------------------------
# drawn cases
# ------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A feature count: usually a multiple of 64 as models have them, sometimes any number."""
    w = _log(rng, lo, hi)
    return max(64, w // 64 * 64) if w >= 64 and rng.random() < 0.65 else w


_DRAWN_KINDS = ("mlp_step", "gpt2_step", "dense", "dense", "dense", "dense", "norm", "embedding", "conv2d",
                "gradproj", "gradproj", "gradproj_embedding", "similarity")
# a drawn case stays under the largest listed one: tensor work, fp32 as the three products it takes,
# and bytes
_MOST_FLOPS = 3.5e12
_MOST_BYTES = 1.2e9


def draw(rng):
    while True:
        case = _draw_kind(rng, rng.choice(_DRAWN_KINDS))
        w = work(case)
        if w["flops"] * (3 if case["dtype"] == "fp32" else 1) <= _MOST_FLOPS and w["bytes"] <= _MOST_BYTES:
            return case


def _draw_kind(rng, kind):
    dtype = "bf16" if rng.random() < 0.6 else "fp32"
    case = {"kind": kind, "dtype": dtype}
    if kind == "mlp_step":
        case.update(n_train=_log(rng, 4, 256), n_val=_log(rng, 1, 32), d_in=_width(rng, 16, 2048),
                    hidden=_width(rng, 32, 2048), d_out=_log(rng, 2, 1000))
    elif kind == "gpt2_step":
        case.update(dtype="bf16", n_train=_log(rng, 1, 16), n_val=_log(rng, 1, 4), T=_log(rng, 16, 1024),
                    layers=rng.randint(1, 4), d=64 * rng.randint(2, 12), vocab=_log(rng, 500, 50257))
    elif kind == "dense":
        wide = rng.random() < 0.15
        layer = rng.choice(("linear", "conv1d"))
        case.update(layer=layer, bias=layer == "conv1d" or rng.random() < 0.5,
                    n_train=_log(rng, 1, 256 if dtype == "bf16" else 64), n_val=_log(rng, 1, 32 if dtype == "bf16" else 16),
                    T=_log(rng, 1, 2048), d_in=_width(rng, 32, 4096 if dtype == "bf16" else 2048),
                    d_out=_width(rng, 4096, 50304) if wide and dtype == "bf16" else _width(rng, 32, 4096 if dtype == "bf16" else 2048))
    elif kind == "norm":
        case.update(rms=rng.random() < 0.5, n_train=_log(rng, 1, 64), n_val=_log(rng, 1, 16), T=_log(rng, 1, 4096),
                    d=_width(rng, 64, 8192))
    elif kind == "embedding":
        case.update(ids=rng.choice(("text", "uniform", "position")), n_train=_log(rng, 1, 64), n_val=_log(rng, 1, 16),
                    T=_log(rng, 16, 2048), d=_width(rng, 64, 2048), vocab=_log(rng, 500, 50304))
        if case["ids"] == "position":
            case["vocab"] = max(case["T"], min(case["vocab"], 4096))
    elif kind == "conv2d":
        case.update(bias=rng.random() < 0.5, n_train=_log(rng, 2, 128), n_val=_log(rng, 1, 16), side=_log(rng, 7, 56),
                    c_in=_log(rng, 3, 256), c_out=_log(rng, 8, 256), k=rng.choice((1, 3, 3, 5)), stride=rng.choice((1, 1, 2)))
        d = case["c_in"] * case["k"] ** 2
        side = _conv_side(case)
        if (case["n_train"] + case["n_val"]) * side * side * d > 1.5e8 or d * case["c_out"] > 4e6:
            return _draw_kind(rng, kind)
    elif kind == "gradproj":
        k = _log(rng, 4, 64)
        case.update(layer=rng.choice(("linear", "linear", "conv1d")), batch=_log(rng, 1, 32), T=_log(rng, 1, 4096),
                    d_in=_width(rng, 64, 14336), d_out=_width(rng, 64, 14336), k_i=k, k_o=k)
        if rng.random() < 0.4:
            case["k_i"] = max(1, k // 2)
    elif kind == "gradproj_embedding":
        k = _log(rng, 4, 64)
        case.update(ids=rng.choice(("text", "uniform")), batch=_log(rng, 1, 32), T=_log(rng, 16, 4096),
                    d=_width(rng, 64, 4096), vocab=_log(rng, 500, 50304), k_i=k, k_o=k)
    else:
        case.update(n1=_log(rng, 1, 128), n2=_log(rng, 1, 512), dim=_log(rng, 256, 1 << 20))
    return case


def _conv_side(case):
    return (case["side"] + 2 * (case["k"] // 2) - case["k"]) // case["stride"] + 1


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _activations(shape, gen, dtype):
    """Layer inputs: unit variance around a mean of each feature's own, as after a norm and a bias."""
    x = torch.randn(shape, generator=gen, device="cuda")
    x += 0.25 * torch.randn(shape[-1], generator=gen, device="cuda")
    return x.to(dtype)


def _out_grads(shape, gen, dtype):
    """Gradients of a mean loss over all tokens: a common direction under the noise, small values."""
    rows = max(1, math.prod(shape[:-1]))
    x = torch.randn(shape, generator=gen, device="cuda")
    x += 0.1 * torch.randn(shape[-1], generator=gen, device="cuda")
    return (x / rows).to(dtype)


def _token_ids(shape, vocab, pattern, gen):
    if pattern == "position":
        return torch.arange(shape[1], device="cuda").expand(shape).contiguous()
    if pattern == "uniform":
        return torch.randint(0, vocab, shape, generator=gen, device="cuda")
    # text: frequency falls with the rank, the most frequent id takes about 4 percent
    weights = 1.0 / (torch.arange(vocab, device="cuda", dtype=torch.float64) + 2.5)
    edges = torch.cumsum(weights, 0)
    u = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * edges[-1]
    rank = torch.searchsorted(edges, u).clamp_(max=vocab - 1)
    return torch.randperm(vocab, generator=gen, device="cuda")[rank]


def _conv1d(d_in, d_out):
    from transformers.pytorch_utils import Conv1D
    return Conv1D(d_out, d_in)          # has a bias always


class _RMSNorm(nn.Module):
    """Llama-style norm: the class name and the 1-D weight are what the hook registration goes by."""

    def __init__(self, d):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(d))
        self.variance_epsilon = 1e-6


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], _DT[case["dtype"]]
    state = {"kind": kind}
    if kind in ("mlp_step", "gpt2_step"):
        with torch.random.fork_rng(devices=[0]), torch.device("cuda"):
            torch.manual_seed(seed)
            if kind == "mlp_step":
                model = make_mlp(case["d_in"], case["hidden"], case["d_out"])
            else:
                model = GPT2Like(GPT2Config(vocab_size=case["vocab"], n_positions=case["T"], n_embd=case["d"],
                                            n_layer=case["layers"], n_head=case["d"] // 64))
        model = model.to("cuda", dtype)
        n = case["n_train"] + case["n_val"]
        if kind == "mlp_step":
            x = torch.randn((n, case["d_in"]), generator=gen, device="cuda").to(dtype)
            y = torch.randint(0, case["d_out"], (n,), generator=gen, device="cuda")
        else:
            x = y = torch.randint(0, case["vocab"], (n, case["T"]), generator=gen, device="cuda")
        engine = GradDotProdEngine(module=model, val_batch_size=case["n_val"], loss_reduction="mean",
                                   use_dummy_bias=kind == "gpt2_step")
        engine.attach(torch.optim.SGD(model.parameters(), lr=0.1))
        state.update(model=model, engine=engine, x=x, y=y, n_train=case["n_train"])
        return state
    if kind == "similarity":
        state["a"] = torch.randn((case["n1"], case["dim"]), generator=gen, device="cuda").to(dtype)
        state["b"] = torch.randn((case["n2"], case["dim"]), generator=gen, device="cuda").to(dtype)
        # two blocks of gradients of one model are not independent
        state["b"][:, ::7] += state["a"][0, ::7]
        return state
    if kind in ("gradproj", "gradproj_embedding"):
        batch, T = case["batch"], case["T"]
        with torch.device("cuda"):
            if kind == "gradproj_embedding":
                layer, d_in, d_out = nn.Embedding(case["vocab"], case["d"]), case["vocab"], case["d"]
                inp = _token_ids((batch, T), case["vocab"], case["ids"], gen)
            else:
                d_in, d_out = case["d_in"], case["d_out"]
                layer = nn.Linear(d_in, d_out, bias=False) if case["layer"] == "linear" else _conv1d(d_in, d_out)
                inp = _activations((batch, T, d_in), gen, dtype)
        grad = _out_grads((batch, T, d_out), gen, dtype)
        # of a Conv1D, P_i projects the out-grad and P_o the activations
        n_i, n_o = (d_out, d_in) if case.get("layer") == "conv1d" else (d_in, d_out)
        P_i = init_projection_matrix_gaussian(case["k_i"], n_i, device="cuda", seed=seed)
        P_o = init_projection_matrix_gaussian(case["k_o"], n_o, device="cuda", seed=seed + 1000)
        state.update(layer=layer.to(dtype), hooks=create_projection_hooks(layer, "layer", P_i, P_o), inp=inp, grad=grad)
        return state
    # one hooked layer and the pair its backward hook gets
    n, n_val = case["n_train"] + case["n_val"], case["n_val"]
    with torch.device("cuda"):
        if kind == "dense":
            d_in, d_out = case["d_in"], case["d_out"]
            layer = nn.Linear(d_in, d_out, bias=case["bias"]) if case["layer"] == "linear" else _conv1d(d_in, d_out)
            lead = (n, case["T"]) if case["T"] > 1 else (n,)
            inp, grad = _activations(lead + (d_in,), gen, dtype), _out_grads(lead + (d_out,), gen, dtype)
        elif kind == "norm":
            layer = _RMSNorm(case["d"]) if case["rms"] else nn.LayerNorm(case["d"])
            layers.maybe_register_rmsnorm(type(layer))
            inp = _activations((n, case["T"], case["d"]), gen, dtype)
            grad = _out_grads((n, case["T"], case["d"]), gen, dtype)
        elif kind == "embedding":
            layer = nn.Embedding(case["vocab"], case["d"])
            inp = _token_ids((n, case["T"]), case["vocab"], case["ids"], gen)
            grad = _out_grads((n, case["T"], case["d"]), gen, dtype)
        else:
            layer = nn.Conv2d(case["c_in"], case["c_out"], case["k"], stride=case["stride"], padding=case["k"] // 2,
                              bias=case["bias"])
            side = _conv_side(case)
            inp = torch.relu(torch.randn((n, case["c_in"], case["side"], case["side"]), generator=gen, device="cuda")).to(dtype)
            grad = (torch.randn((n, case["c_out"], side, side), generator=gen, device="cuda") / n).to(dtype)
    state.update(layer=layer.to(dtype), inp=inp, grad=grad, n_val=n_val)
    return state


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("mlp_step", "gpt2_step"):
        return _run_step(state)
    if kind == "similarity":
        return projection_similarity(state["a"], state["b"])
    if kind in ("gradproj", "gradproj_embedding"):
        layer, h = state["layer"], state["hooks"]
        h.forward_hook_store_inputs(layer, (state["inp"],), None)
        h.backward_hook_compute_proj(layer, None, (state["grad"],))
        return layer._ghost_grad_proj
    layer, n_val = state["layer"], state["n_val"]
    hooks._capture_activations(layer, (state["inp"],), None)
    layers.begin_deferred_dots()
    hooks._prepare_sample_grad_or_dotprod(layer, (state["grad"],), n_val, "mean")
    hooks._apply_train_grad(layer, n_val, "mean")
    layers.finalize_pending_dots()
    out = {}
    for name, p in layer.named_parameters():
        out[name] = (p.grad_dot_prod, p.grad_dot_prod_matrix, p.train_grad)
        del p.grad_dot_prod, p.grad_dot_prod_matrix, p.train_grad
    return out


def _run_step(state):
    model, engine, x, y, n_train = (state[k] for k in ("model", "engine", "x", "y", "n_train"))
    engine.attach_train_batch(x[:n_train], y[:n_train], 0, 0)
    if state["kind"] == "mlp_step":
        loss = nn.functional.cross_entropy(model(x), y)
    else:
        loss, _ = model(x, labels=y)
    loss.backward()
    engine.prepare_gradients()
    engine.aggregate_and_log()
    logged = engine.dot_product_log.pop()
    engine.clear_gradients()
    out = {"loss": loss.detach(), "vector": logged["dot_product"], "matrix": logged["dot_product_matrix"]}
    for name, p in model.named_parameters():
        if "dummy_bias" not in name:
            out[name] = p.grad
    model.zero_grad(set_to_none=True)
    return out


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _dense_flops(n_t, n_v, T, d, p):
    """Dot products of all pairs and the train gradient, by the cheaper of the two ways: token Grams
    of the pairs and one GEMM, or every sample's gradient (whose sum is the train gradient)."""
    gram = 2.0 * n_t * n_v * T * T * (d + p) + 2.0 * n_t * T * d * p
    per_sample = 2.0 * (n_t + n_v) * T * d * p + 2.0 * n_t * n_v * d * p
    return min(gram, per_sample)


def work(case):
    kind, s = case["kind"], _SIZE[case["dtype"]]
    if kind == "similarity":
        n1, n2, dim = case["n1"], case["n2"], case["dim"]
        return {"bytes": s * (n1 + n2) * dim + 4 * n1 * n2, "flops": 2.0 * n1 * n2 * dim}
    if kind == "gradproj":
        rows, d, p, ki, ko = case["batch"] * case["T"], case["d_in"], case["d_out"], case["k_i"], case["k_o"]
        a, b = (ko, ki) if case["layer"] == "conv1d" else (ki, ko)
        return {"bytes": s * rows * (d + p) + 4 * (a * d + b * p) + 4 * case["batch"] * ki * ko,
                "flops": 2.0 * rows * (d * a + p * b + ki * ko)}
    if kind == "gradproj_embedding":
        rows, d, ki, ko = case["batch"] * case["T"], case["d"], case["k_i"], case["k_o"]
        table = min(rows, case["vocab"])
        return {"bytes": rows * (s * d + 8) + 4 * ki * table + 4 * ko * d + 4 * case["batch"] * ki * ko,
                "flops": 2.0 * rows * (d * ko + ki * ko)}
    n_t, n_v = case["n_train"], case["n_val"]
    n = n_t + n_v
    if kind == "mlp_step":
        dims = [(case["d_in"], case["hidden"]), (case["hidden"], case["hidden"]), (case["hidden"], case["d_out"])]
        flops = sum(4.0 * n * d * p + _dense_flops(n_t, n_v, 1, d, p) for d, p in dims) - 2.0 * n * dims[0][0] * dims[0][1]
        return {"bytes": sum(3 * s * d * p + 4 * s * n * (d + p) for d, p in dims), "flops": flops}
    if kind == "gpt2_step":
        T, d, L, V = case["T"], case["d"], case["layers"], (case["vocab"] + 63) // 64 * 64
        dims = [(d, 3 * d), (d, d), (d, 4 * d), (4 * d, d)] * L + [(d, V)]
        flops = sum(4.0 * n * T * a * b + _dense_flops(n_t, n_v, T, a, b) for a, b in dims) + L * 6.0 * n * T * T * d
        return {"bytes": sum(3 * s * a * b + 3 * s * n * T * (a + b) for a, b in dims), "flops": flops}
    if kind == "norm":
        params = 1 if case["rms"] else 2
        return {"bytes": 2 * s * n * case["T"] * case["d"] + params * (s * case["d"] + 4 * n_v * n_t),
                "flops": 8.0 * n * case["T"] * case["d"]}
    if kind == "embedding":
        return {"bytes": n * case["T"] * (s * case["d"] + 8) + s * case["vocab"] * case["d"] + 4 * n_v * n_t,
                "flops": 1.0 * n * case["T"] * case["d"]}
    if kind == "conv2d":
        side = _conv_side(case)
        T, d, p = side * side, case["c_in"] * case["k"] ** 2, case["c_out"]
        moved = s * n * (case["c_in"] * case["side"] ** 2 + T * p)
    else:
        T, d, p = case["T"], case["d_in"], case["d_out"]
        moved = s * n * T * (d + p)
    return {"bytes": moved + s * d * p + 4 * n_v * n_t, "flops": _dense_flops(n_t, n_v, T, d, p)}


def tolerance(case):
    if case["kind"] == "gpt2_step":
        return {"rel": 2e-2}         # a bf16 model pass before the compared products
    if case["kind"] == "similarity":
        return {"rel": 3e-5}         # exact products of the given values, 32-bit sums
    # bf16 operands and stored intermediates; fp32 operands carried as two bf16 parts each (16 bits)
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 3e-5}
