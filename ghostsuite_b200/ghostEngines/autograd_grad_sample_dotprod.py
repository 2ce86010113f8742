"""Forward/backward hook plumbing for the gradient-dot-product engine.

Drop-in for GhostSuite's ``ghostEngines/autograd_grad_sample_dotprod.py`` (``add_hooks`` :23-81,
``remove_hooks`` :84-89, ``_capture_activations`` :92-94, ``backward_hook`` closure :58-71): same
names, signatures, attributes (``layer.activations``, ``layer.backprops``, ``layer.name``,
``model.autograd_grad_sample_hooks``) and exceptions.  The hook bodies call the CUDA-backed layer
functions of ``supported_layers_grad_samplers_dotprod``.

One deliberate difference inside the hook: the reference multiplies the whole out-grad tensor by
the batch size (a full extra read and write per layer, :132-134) before the train-gradient pass.
Here the raw out-grad is kept and the factor is recorded in ``layer._ghost_backprop_scale``; the
kernels fold it into their epilogue scale.
"""
from __future__ import annotations

import weakref
from typing import Tuple

import torch
import torch.nn as nn

from .. import _lib, ops
from . import supported_layers_grad_samplers_dotprod as _layers
from .supported_layers_grad_samplers_dotprod import (
    _param,
    _wanted,
    _supported_layers_dotprod,
    _create_or_accumulate_train_grad,
)


#: optional ``fn(layer, A, B, n_val_local) -> (A_full, B_full, n_val_global)`` applied to every hooked
#: layer's operands before its layer functions run.  The data-parallel layer installs one when the
#: validation batch is split over ranks: it appends the other ranks' validation rows (an all-gather
#: into local memory), so the kernels see ``cat(train_local, val_global)`` without every rank having
#: run the whole validation batch through the model.
VALIDATION_GATHER = None


def requires_grad(module: nn.Module) -> bool:
    """True if any parameter of ``module`` was trainable when the engine was built."""
    return any(getattr(p, "initially_requires_grad", p.requires_grad) for p in module.parameters())


def add_hooks(model: nn.Module, val_batch_size: int, loss_reduction: str = "mean"):
    """Register the activation-capture and dot-product/train-gradient hooks on every supported
    layer that has a trainable parameter.  Calling it twice on one model raises ValueError."""
    if hasattr(model, "autograd_grad_sample_hooks"):
        raise ValueError("Trying to add hooks twice to the same model")
    if loss_reduction not in ("mean", "sum"):
        raise ValueError(f"loss_reduction must be 'mean' or 'sum', got {loss_reduction!r}")

    handles = []
    for name, layer in model.named_modules():
        if type(layer) not in _supported_layers_dotprod and getattr(layer, "weight", None) is not None \
                and layer.weight.dim() == 1:
            _layers.maybe_register_rmsnorm(type(layer))
        if type(layer) in _supported_layers_dotprod and requires_grad(layer):
            layer.name = name

            def backward_hook(this_layer, grad_input, grad_output):
                _prepare_sample_grad_or_dotprod(this_layer, grad_output, val_batch_size, loss_reduction)
                _apply_train_grad(this_layer, val_batch_size)
                return None

            handles.extend(register_hook_pair(layer, _capture_activations, backward_hook, "activations"))
        elif not list(layer.children()) and requires_grad(layer):
            print(f"WARNING: Skipping atomic layer '{name}' of type {type(layer)} because it is not supported.")

    model.__dict__.setdefault("autograd_grad_sample_hooks", []).extend(handles)


def register_hook_pair(layer: nn.Module, capture, backward_hook, slot: str):
    """Register ``capture(layer, inputs, outputs)``, which keeps the input as attribute ``slot``, on the
    forward pass and ``backward_hook(layer, grad_input, (grad,))`` on the output's gradient; returns the
    removable handles.

    The backward hooks read the output gradient only, so a hook on the autograd node that produced the
    output serves them; a module's full backward hook wraps input and output in two more nodes per call
    (about 60 us of host time per layer and step).  On the node, like there, the gradient is what the
    hooks that a user has put on the output tensor leave of it, and ``autograd.grad`` up to the output
    calls nothing.  Embeddings keep the module hook: their input has no gradient, in which case a module
    hook that a user registers after this one fires at the output too, and would come before a hook on
    the node inside.

    Every call's backward hook gets the input of that call.  Of calls that follow each other without
    a backward pass in between only the last may be differentiated, as with one slot per layer; a
    recomputation inside the backward pass (activation checkpointing) makes room for one more."""
    if isinstance(layer, nn.Embedding):
        return [layer.register_forward_hook(capture), layer.register_full_backward_hook(backward_hook)]

    due = slot + "_due"

    def forward_hook(layer, inputs, outputs):
        if torch._C._get_tracing_state() is not None:
            # as torch says of full backward hooks: the trace would run on without them
            raise ValueError(f"Modules that have backward hooks assigned can't be compiled: {layer}")
        capture(layer, inputs, outputs)
        out = outputs if torch.is_tensor(outputs) else next((o for o in outputs if torch.is_tensor(o)), None)
        if out is None or not out.requires_grad or not torch.is_grad_enabled():
            return
        own = layer.__dict__
        own[due] = True
        # The graph holds what follows, and the collector does not look into it: the layer is held weakly (it may
        # hold the graph), and the input in a list that the hook empties (a graph may outlive its backward pass).
        ref, kept = weakref.ref(layer), [own.get(slot)]
        if torch._C._current_graph_task_id() != -1:
            own.pop(slot, None)          # recomputed: no hook may follow that would clear it

        def on_gradient(grad):
            value, layer = kept.pop() if kept else None, ref()
            if layer is None:
                return
            own = layer.__dict__
            own[slot] = value if own.pop(due, False) else None
            backward_hook(layer, None, (grad,))

        _hook_output(out, on_gradient)

    return [layer.register_forward_hook(forward_hook)]


def _hook_output(out: torch.Tensor, fn) -> None:
    """``fn(gradient)`` when the node that hands on the gradient of ``out`` is about to run.  Linear layers return a
    reshaped view of their product; an in-place operation on a view gives it a new node and drops the old
    one with its hooks, so there the base's node is taken.  The native form of this saves 5 us of host
    time per layer and step; the compiler traces the one here."""
    if _lib.binding_present() and not torch.compiler.is_compiling():
        if not _lib.native().hook_output(out, fn):
            out.register_hook(fn)           # a leaf handed through (a layer that returns its parameter)
        return
    node, index, shape = out.grad_fn, out.output_nr, out.shape
    if out._is_view():
        base = out._base
        if base.requires_grad and base.grad_fn is not None and base.numel() == out.numel() \
                and base.is_contiguous() and out.is_contiguous():
            node, index = base.grad_fn, base.output_nr
    if node is None:
        out.register_hook(fn)
        return

    def on_gradients(grads):
        grad = grads[index]
        fn(grad if grad is None or grad.shape == shape else grad.reshape(shape))

    node.register_prehook(on_gradients)


def remove_hooks(model: nn.Module):
    """Remove everything ``add_hooks`` registered."""
    _layers.finalize_pending_dots()
    if hasattr(model, "autograd_grad_sample_hooks"):
        for handle in model.autograd_grad_sample_hooks:
            handle.remove()
        del model.autograd_grad_sample_hooks


def _capture_activations(layer: nn.Module, inputs: Tuple, outputs: Tuple):
    """Forward hook: keep the layer input for the backward hook.  A forward without autograd
    (evaluation, or the first pass of re-entrant activation checkpointing) is followed by no
    backward hook and keeps nothing alive."""
    if not torch.is_grad_enabled():
        return
    layer.__dict__["activations"] = inputs[0].detach()


def _prepare_sample_grad_or_dotprod(layer: nn.Module, grad_output: Tuple[torch.Tensor],
                                    val_batch_size: int, loss_reduction: str = "mean"):
    """Backward hook, part 1: dot products of this layer's parameters (reference :97-137)."""
    backprops = grad_output[0]
    if backprops.requires_grad:
        backprops = backprops.detach()
    # instance attributes are written to the dictionary: nn.Module.__setattr__ searches the parameter,
    # buffer and module tables for each of these names first
    own = layer.__dict__
    A = own.setdefault("activations", None)
    dot_fn, _ = _supported_layers_dotprod[type(layer)]

    # mixed precision: bring both operands to the common floating type (ids stay integer)
    if A is not None and A.dtype is not backprops.dtype and A.is_floating_point():
        common = torch.promote_types(A.dtype, backprops.dtype)
        A = A.to(common)
        backprops = backprops.to(common)
        own["activations"] = A

    # 'mean' losses carry a 1/batch factor (the batch this process ran); the train-gradient kernels
    # undo it in their epilogue
    own["_ghost_backprop_scale"] = float(backprops.shape[0]) if loss_reduction == "mean" else 1.0
    # the per-parameter [n_train] vectors are reduced in one batched op when the backward pass ends
    if _layers._PENDING_DOTS is None and _layers.begin_deferred_dots():
        try:
            torch.autograd.Variable._execution_engine.queue_callback(_layers.finalize_pending_dots)
        except Exception:
            _layers.finalize_pending_dots()      # not inside a backward pass: reduce immediately
    exchange = _layers.VALIDATION_EXCHANGE
    if exchange is not None and VALIDATION_GATHER is not None and A is not None and A.is_floating_point():
        # validation batch split over ranks: the ranks exchange validation gradients where the layer
        # type allows it ...
        own["_ghost_val_batch"] = val_batch_size
        try:
            handled = _layers.dot_product_with_exchange(layer, A, backprops, val_batch_size, exchange)
        except BaseException:
            _layers.finalize_pending_dots()
            raise
        if handled:
            own["backprops"] = backprops
            return
    if VALIDATION_GATHER is not None and A is not None:
        # ... and validation operands everywhere else
        A, backprops, val_batch_size = VALIDATION_GATHER(layer, A, backprops, val_batch_size)
        own["activations"] = A
    own["_ghost_val_batch"] = val_batch_size
    try:
        dot_fn(layer, A, backprops, val_batch_size=val_batch_size)
    except BaseException:
        _layers.finalize_pending_dots()          # a failed pass may never reach its callback
        raise
    own["backprops"] = backprops


_PASS_ATTRIBUTES = ("activations", "backprops", "_ghost_backprop_scale", "_ghost_val_batch", "_ghost_colsums",
                    "_ghost_bias_grad", "_ghost_jobs", "_ghost_norm_grads", "_ghost_cached_train_grad", "_ghost_ln_cache", "_ghost_conv_tokens")


def _apply_train_grad(layer: nn.Module, val_batch_size: int, loss_reduction: str = "mean"):
    """Backward hook, part 2: averaged train gradients into ``param.train_grad`` (reference :140-196)."""
    own, kind = layer.__dict__, type(layer)
    _, train_grad_fn = _supported_layers_dotprod.get(kind, (None, None))
    val_batch_size = own.get("_ghost_val_batch", val_batch_size)
    if not train_grad_fn:
        raise ValueError(
            f"Layer {layer.__class__.__name__} is not supported for training gradient computation. "
            "Ensure it is included in the _supported_layers_dotprod dictionary.")
    try:
        if kind in _layers._SELF_APPLYING or isinstance(layer, nn.LayerNorm):
            train_grad_fn(layer, layer.activations, layer.backprops, val_batch_size)
        else:
            weight, bias = _param(layer, "weight"), _param(layer, "bias")
            if weight is not None and _wanted(weight, weight.requires_grad):
                grad_weight = train_grad_fn(layer, layer.activations, layer.backprops, val_batch_size)
                if grad_weight is None:
                    raise ValueError(
                        f"Layer {layer.__class__.__name__} returned None for weight gradient. "
                        "Ensure the compute_layer_train_grad function is implemented correctly.")
                if grad_weight is not _layers.DEFERRED:      # else: handed over by the launch that makes it
                    _create_or_accumulate_train_grad(weight, grad_weight)
            if bias is not None and _wanted(bias, bias.requires_grad):
                _train_grad_bias_from_layer(layer, val_batch_size, loss_reduction)
    finally:
        for attr in _PASS_ATTRIBUTES:
            own.pop(attr, None)


def _train_grad_bias_from_layer(layer: nn.Module, val_batch_size: int, loss_reduction: str) -> None:
    """Bias train gradient from the per-sample column sums the dot-product pass already made, added to
    ``layer.bias.train_grad`` (inside a backward pass: by the batched launch at its end)."""
    B = layer.backprops
    n_train = B.size(0) - val_batch_size
    if n_train <= 0:
        raise ValueError("No training samples to compute gradients, check batch sizes.")
    own = layer.__dict__
    colsums = own.get("_ghost_colsums")
    if colsums is None:
        if isinstance(layer, nn.Conv2d):      # features are dim 1 there: [N, p, H, W] -> [N, H*W, p]
            B = B.reshape(B.size(0), B.size(1), -1).transpose(1, 2).contiguous()
        colsums = ops.colsum(B)
    scale = float(getattr(layer, "_ghost_backprop_scale", 1.0))
    if loss_reduction == "mean":
        scale /= n_train
    bias = _param(layer, "bias")
    if _layers._sum_into_job(own, bias, colsums, n_train, scale, own.get("_ghost_bias_grad")):
        return
    out_dtype = torch.bfloat16 if bias.dtype is torch.bfloat16 else torch.float32
    _layers._train_grad_from_vectors(bias, colsums, n_train, scale, out_dtype, own.get("_ghost_bias_grad"))


def _compute_train_grad_bias(B: torch.Tensor, val_batch_size: int, loss_reduction: str = "mean") -> torch.Tensor:
    """Sum (or, for 'mean', average over the train samples) of the already scaled out-grad over
    batch and tokens -> ``[features]`` (reference :199-222)."""
    n_train = B.size(0) - val_batch_size
    if n_train <= 0:
        raise ValueError("No training samples to compute gradients, check batch sizes.")
    colsums = ops.colsum(B)
    out_dtype = B.dtype if B.dtype in (torch.float32, torch.bfloat16) else torch.float32
    return ops.rows_sum(colsums, n_train, 1.0 / n_train if loss_reduction == "mean" else 1.0, out_dtype)
