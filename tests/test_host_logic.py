"""Host-side logic that needs no GPU: deferred reduction of the dot-product vectors, the path rule's
cost model, the flat projection file format."""
import contextlib
import inspect
import io
import os

import numpy as np
import pytest
import torch
from torch import nn

from ghostsuite_b200.ghostEngines import supported_layers_grad_samplers_dotprod as L


def test_deferred_dot_vectors_are_reduced_in_one_batch():
    params = [nn.Parameter(torch.zeros(3)) for _ in range(3)]
    mats = [torch.randn(4, 6) for _ in range(4)]
    assert L.begin_deferred_dots() is True
    assert L.begin_deferred_dots() is False              # already collecting
    L._set_dot(params[0], mats[0])
    L._set_dot(params[1], mats[1])
    L._set_dot(params[2], mats[2])
    L._set_dot(params[0], mats[3])                        # a tied parameter: the last hook wins
    assert params[1].grad_dot_prod_matrix is mats[1]
    L.finalize_pending_dots()
    for p, m in zip(params, (mats[3], mats[1], mats[2])):
        assert p.grad_dot_prod_matrix is m
        assert p.grad_dot_prod.shape == (6,)
        assert torch.allclose(p.grad_dot_prod, m.sum(0))
    L.finalize_pending_dots()                             # nothing pending: a no-op
    q = nn.Parameter(torch.zeros(1))
    L._set_dot(q, mats[0])                                # outside a backward pass: reduced at once
    assert torch.allclose(q.grad_dot_prod, mats[0].sum(0))


def _decide(n_t, n_v, T, d, p, rule="cost", dtype=torch.bfloat16):
    layer = nn.Linear(d, p, bias=False, device="meta")
    A = torch.empty(n_t + n_v, T, d, dtype=dtype, device="meta")
    B = torch.empty(n_t + n_v, T, p, dtype=dtype, device="meta")
    old = L.PATH_RULE
    L.PATH_RULE = rule
    try:
        L._should_use_ghost_computation(layer, A, B, val_batch_size=n_v)
    finally:
        L.PATH_RULE = old
    return layer.use_ghost_computation


def test_path_rule_follows_the_measured_crossover():
    # single layer 4096 -> 11008: the Gram kernel wins at T = 128, the per-sample path from T = 512 on
    assert _decide(256, 32, 128, 4096, 11008) is True
    assert _decide(256, 32, 512, 4096, 11008) is False
    assert _decide(64, 8, 2048, 4096, 11008) is False
    assert _decide(16, 2, 8192, 4096, 11008) is False
    # GPT-2 layers at T = 1024 take the per-sample path, the T = 1 MLP the Gram kernel
    for d, p in ((768, 2304), (768, 768), (768, 3072), (3072, 768), (768, 50304)):
        assert _decide(32, 8, 1024, d, p) is False
    assert _decide(64, 16, 1, 512, 1024, dtype=torch.float32) is True
    # the reference's rule 2 T^2 <= numel and the forced rules
    assert _decide(32, 8, 1024, 768, 2304, rule="reference") is False        # 2 * 1024^2 > 1.77 M
    assert _decide(32, 8, 1024, 768, 3072, rule="reference") is True         # 2 * 1024^2 <= 2.36 M
    assert _decide(32, 8, 1024, 768, 50304, rule="reference") is True
    assert _decide(32, 8, 1024, 768, 768, rule="gram") is True
    assert _decide(256, 32, 128, 4096, 11008, rule="persample") is False


def test_flat_projection_file_round_trip(tmp_path):
    from ghostsuite_b200.ghostEngines.gradProjection.gradproj_engine import GradProjLoraEngine, load_projection_bin
    torch.manual_seed(0)
    model = nn.Sequential(nn.Linear(10, 24), nn.ReLU(), nn.Linear(24, 5))
    with contextlib.redirect_stdout(io.StringIO()):
        eng = GradProjLoraEngine(model, "0,2", 16, 2, 42, "float32", str(tmp_path / "p"), proj_format="bin")
    rows = [torch.randn(n, eng.total_proj_dim) for n in (4, 3, 5)]
    for it, r in enumerate(rows):
        eng.iteration = it
        with contextlib.redirect_stdout(io.StringIO()):
            eng._save_projection(r, batch_indices=list(range(100 * it, 100 * it + r.shape[0])))
    eng.flush()
    data, index = load_projection_bin(str(tmp_path / "p"))
    assert data.shape == (12, eng.total_proj_dim) and index["dtype"] == "float32"
    assert [b["row0"] for b in index["batches"]] == [0, 4, 7]
    assert index["batches"][2]["batch_idx"] == [200, 201, 202, 203, 204]
    assert np.array_equal(np.asarray(data), torch.cat(rows).numpy())
    eng.cleanup()


def test_choose_ki_ko_reproduces_the_reference_table(golden):
    """``choose_ki_ko`` against the (n_i, n_o, k_total, k_min) -> (k_i, k_o) rows that the golden
    script recorded from the reference's projection_utils.choose_ki_ko (:12-66 there)."""
    from ghostsuite_b200.ghostEngines.gradProjection.projection_utils import choose_ki_ko
    table = golden["choose_ki_ko_table"]
    assert table.shape[0] >= 7
    for n_i, n_o, k_total, k_min, k_i, k_o in table.tolist():
        assert choose_ki_ko(n_i, n_o, k_total, k_min) == (k_i, k_o), (n_i, n_o, k_total, k_min)


def test_parameter_walk_of_modules_with_tables_of_their_own():
    """Wrappers that rename their parameters, scripted modules and shared parameters: as torch lists them."""
    from ghostsuite_b200 import _lib

    class Renaming(nn.Module):
        def __init__(self):
            super().__init__()
            self.inner = nn.Linear(2, 2)

        def named_parameters(self, *args, **kwargs):
            for name, p in super().named_parameters(*args, **kwargs):
                yield name.replace("inner.", ""), p

    tied = nn.Sequential(nn.Linear(2, 2), nn.Linear(2, 2))
    tied[1].weight = tied[0].weight
    for m in (Renaming(), torch.jit.script(nn.Linear(2, 2)), nn.Sequential(torch.jit.script(nn.Linear(2, 2))), tied):
        want, got = list(m.named_parameters()), _lib.named_parameters(m)
        assert [n for n, _ in got] == [n for n, _ in want]
        assert all(a.data_ptr() == b.data_ptr() for (_, a), (_, b) in zip(got, want))


_DENSE_HOOK = inspect.signature(L.ops.dense_hook)


def _hook_arguments(monkeypatch, layer, dtype=torch.float32, n=6, n_val=2):
    """What the backward hook of a dense layer asks the native call for."""
    seen = {}

    def call(*args, **kwargs):
        bound = _DENSE_HOOK.bind(*args, **kwargs)
        bound.apply_defaults()
        seen.update(bound.arguments)
        return torch.zeros(n_val, n - n_val), None, None, torch.zeros(n_val, n - n_val), None

    monkeypatch.setattr(L.ops, "dense_hook", call)
    monkeypatch.setattr(L, "_gram_of_vectors", lambda X, n_v, M=None: M)
    layer._ghost_backprop_scale = 1.0
    L._compute_linear_dot_product(layer, torch.zeros(n, layer.in_features, dtype=dtype),
                                  torch.zeros(n, layer.out_features, dtype=dtype), n_val)
    del layer._ghost_backprop_scale
    return seen


def test_switch_for_fused_column_sums_reaches_the_hook(monkeypatch):
    assert _hook_arguments(monkeypatch, nn.Linear(8, 8))["fuse_colsums"] is True
    monkeypatch.setattr(L, "FUSE_BIAS_COLSUMS", False)
    assert _hook_arguments(monkeypatch, nn.Linear(8, 8))["fuse_colsums"] is False


def test_preset_path_is_not_passed_over(monkeypatch):
    """The one-launch kernel of small layers stands in for the rule's choice, not for a user's."""
    ruled = nn.Linear(8, 8)
    assert _hook_arguments(monkeypatch, ruled)["any_path"] is True
    assert _hook_arguments(monkeypatch, ruled)["any_path"] is True          # the cached choice is still the rule's
    for choice in (True, False):
        preset = nn.Linear(8, 8)
        preset.use_ghost_computation = choice
        seen = _hook_arguments(monkeypatch, preset)
        assert seen["any_path"] is False and seen["use_gram"] is choice
    ruled.use_ghost_computation = not ruled.use_ghost_computation
    assert _hook_arguments(monkeypatch, ruled)["any_path"] is False
    monkeypatch.setattr(L, "PATH_RULE", "gram")
    assert _hook_arguments(monkeypatch, nn.Linear(8, 8))["any_path"] is False


def test_type_of_an_unwanted_gradient_does_not_matter():
    """``persample_dot`` without a gradient ignores ``grad_dtype``; here it gets as far as asking for CUDA tensors."""
    X = torch.zeros(3, 2, 8)
    for dtype in (torch.float16, torch.float64):
        with pytest.raises(RuntimeError, match="CUDA"):
            L.ops.persample_dot(X, X, 1, want_grad=False, grad_dtype=dtype)
        with pytest.raises(ValueError, match="unsupported dtype"):
            L.ops.persample_dot(X, X, 1, want_grad=True, grad_dtype=dtype)


class _Listing(nn.Module):
    """A wrapper that lists its modules under names of its own and leaves one out."""

    def __init__(self):
        super().__init__()
        self.inner, self.hidden = nn.Linear(2, 2), nn.Linear(2, 2)

    def named_modules(self, memo=None, prefix="", remove_duplicate=True):
        yield prefix, self
        yield prefix + ".renamed", self.inner


def test_native_parameter_walk_agrees_with_torch():
    from ghostsuite_b200 import _lib
    if not os.path.exists(_lib.BINDING_PATH):
        pytest.skip("the torch binding is not built")
    tied = nn.Sequential(nn.Linear(2, 2), nn.Linear(2, 2), nn.LayerNorm(2))
    tied[1].weight = tied[0].weight
    shared = nn.Sequential(tied[0], nn.ModuleDict({"again": tied[0], "none": nn.Identity()}), nn.TransformerEncoderLayer(4, 2))
    shared.register_parameter("absent", None)
    for m in (tied, shared):                               # walked
        found = _lib.native().named_parameters(m, nn.Module.named_modules)
        assert [(n, id(p)) for n, p in found] == [(n, id(p)) for n, p in m.named_parameters()]
    late = nn.Sequential(nn.Linear(2, 2))
    late[0].named_modules = lambda *args, **kwargs: iter(())
    for m in (_Listing(), nn.Sequential(nn.Linear(2, 2), _Listing()), late):          # torch's to list
        assert _lib.native().named_parameters(m, nn.Module.named_modules) is None
        assert [n for n, _ in _lib.named_parameters(m)] == [n for n, _ in m.named_parameters()]


def test_path_rule_goes_by_the_layout_of_the_weight():
    """A Conv1D d -> p has the tiles of a Linear p -> d, and the same costs otherwise."""
    from transformers.pytorch_utils import Conv1D
    choices = set()
    for n_t, n_v, T in ((64, 1, 32), (64, 1, 100), (24, 5, 60), (24, 5, 197)):
        for d, p in ((300, 1000), (1000, 300), (100, 2000), (768, 768)):
            conv = Conv1D(p, d)
            L._should_use_ghost_computation(conv, torch.empty(n_t + n_v, T, d, device="meta"),
                                            torch.empty(n_t + n_v, T, p, device="meta"), val_batch_size=n_v)
            assert conv.use_ghost_computation is _decide(n_t, n_v, T, p, d, dtype=torch.float32), (n_t, n_v, T, d, p)
            choices.add(conv.use_ghost_computation)
    assert choices == {True, False}


def test_embedding_batch_beyond_one_set_of_buckets(monkeypatch):
    """Train and validation tokens that only together pass 31 bits go through the two separate calls."""
    calls = []
    monkeypatch.setattr(L.ops, "embedding_hook", lambda ids, G, n_val, *a: calls.append("hook") or (torch.zeros(n_val, 3), torch.zeros(4, 8)))
    monkeypatch.setattr(L.ops, "embedding_dot", lambda ids, G, n_val, *a: calls.append("dot") or torch.zeros(n_val, 3))
    monkeypatch.setattr(L.ops, "embedding_wgrad", lambda *a: calls.append("wgrad") or torch.zeros(4, 8))
    layer = nn.Embedding(4, 8)
    layer._ghost_backprop_scale = 1.0
    for T, want in ((2 ** 28, ["hook"]), (2 ** 29, ["dot", "wgrad"])):
        calls.clear()
        A = torch.zeros(1, dtype=torch.long).expand(4, T)
        B = torch.zeros(1).expand(4, T, 8)
        L._compute_embedding_dot_product(layer, A, B, 1)
        L._compute_embedding_train_grad(layer, A, B, 1)
        assert calls == want


@pytest.mark.parametrize("kind", ["linear", "embedding"])
def test_gradproj_hooks_refuse_an_empty_batch(kind):
    """With the error of the reshape that it does not fit, whatever else is missing (here the GPU)."""
    from ghostsuite_b200.ghostEngines.gradProjection.autograd_gradproj import create_projection_hooks
    layer = torch.nn.Linear(6, 4, bias=False) if kind == "linear" else torch.nn.Embedding(6, 4)
    hooks = create_projection_hooks(layer, "layer", torch.randn(2, 6), torch.randn(3, 4))
    inp = torch.zeros(0, 5, 6) if kind == "linear" else torch.zeros(0, 5, dtype=torch.long)
    hooks.forward_hook_store_inputs(layer, (inp,), None)
    with pytest.raises(RuntimeError, match="reshape"):
        hooks.backward_hook_compute_proj(layer, None, (torch.zeros(0, 5, 4),))


def test_large_similarity_sets_that_the_kernel_takes():
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    rows = lambda n, d: torch.zeros(n, d, dtype=torch.bfloat16)
    takes = U._bf16_sets_for_kernel
    assert takes(rows(1, 96), rows(65536, 96)) and takes(rows(129, 101), rows(512, 101))
    assert takes(rows(600, 120)[:, 8:104], rows(3, 96)) and not takes(rows(600, 120)[:, 4:100], rows(3, 96))
    assert not takes(rows(2, 96), rows(65537, 96)) and not takes(rows(513, 101), rows(2, 101))
    assert not takes(rows(200, 95), rows(200, 95)) and not takes(rows(1, 8), rows(200, 8))         # less exact than the GEMM
    assert not takes(rows(0, 96), rows(200, 96)) and not takes(rows(200, 0), rows(200, 0))
    assert not takes(rows(200, 96), rows(200, 96).float()) and not takes(rows(200, 96).double(), rows(200, 96).double())
    assert not takes(rows(1, 96).expand(200, 96), rows(2, 96)) and not takes(rows(96, 200).t(), rows(2, 96))
    assert not takes(rows(200, 96).requires_grad_(), rows(2, 96))
    with torch.autograd.forward_ad.dual_level():
        assert not takes(rows(200, 96), rows(2, 96))
    seen = []
    torch.func.vmap(lambda x: seen.append(takes(x, rows(2, 96))) or x.sum())(torch.zeros(3, 200, 96, dtype=torch.bfloat16))
    assert seen == [False]


def test_large_similarity_sets_that_are_not_plain_rows():
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    a, b = torch.ones(130, 128).bfloat16(), torch.ones(3, 128).bfloat16()
    assert U._bf16_sets_for_kernel(a, b)
    for other in (a.to_sparse(), a.to_sparse_csr(), torch._neg_view(a)):
        assert not U._bf16_sets_for_kernel(other, b) and not U._bf16_sets_for_kernel(b, other)


def test_similarity_of_large_sets_inside_a_dispatch_mode():
    """A mode that follows torch's operations (a trace with real tensors, a counter) does not see the kernel."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    a, b, seen = torch.ones(130, 128).bfloat16(), torch.ones(3, 128).bfloat16(), []

    def scores(x, y):
        seen.append(U._bf16_sets_for_kernel(x, y))
        return U.projection_similarity(x, y)

    traced = make_fx(scores, tracing_mode="real")(a, b)
    assert (traced(2 * a, b) == 256).all()
    with FlopCounterMode(display=False) as count:
        scores(a, b)
    assert count.get_total_flops() == 2 * 130 * 3 * 128
    assert seen == [False, False] and U._bf16_sets_for_kernel(a, b)


@pytest.mark.parametrize("owner,name", [("torch._C", "_get_tracing_state"), ("torch._C._functorch", "peek_interpreter_stack"),
                                        ("torch._C", "_len_torch_dispatch_stack"), ("torch.autograd.forward_ad", "_current_level")])
def test_similarity_without_a_name_of_torch_that_has_no_promise(owner, name, monkeypatch):
    import importlib.util
    import torch.autograd.forward_ad
    from ghostsuite_b200.ghostEngines.gradProjection import projection_utils as U
    holder = torch
    for part in owner.split(".")[1:]:
        holder = getattr(holder, part)
    spec = importlib.util.spec_from_file_location(U.__name__, U.__file__)
    fresh = importlib.util.module_from_spec(spec)
    with monkeypatch.context() as m:
        m.delattr(holder, name)
        spec.loader.exec_module(fresh)
        a, b = torch.ones(130, 128).bfloat16(), torch.ones(3, 128).bfloat16()
        assert not fresh._bf16_sets_for_kernel(a, b)
        assert (fresh.projection_similarity(a, b) == 128).all()
    assert U._bf16_sets_for_kernel(a, b)
