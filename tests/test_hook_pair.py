"""The pair of hooks that both engines put on a layer: which gradient and which input the backward hook
gets.  Its product must be the weight gradient that autograd itself computes."""
import gc
import weakref

import pytest
import torch
import torch.nn.functional as F
from torch import nn
from torch.utils.checkpoint import checkpoint
from transformers.pytorch_utils import Conv1D

from ghostsuite_b200 import _lib
from ghostsuite_b200.ghostEngines.autograd_grad_sample_dotprod import register_hook_pair


@pytest.fixture(autouse=True, params=["native", "python"])
def form(request, monkeypatch):
    """The hook on the node in both its forms."""
    if request.param == "python":
        monkeypatch.setattr(_lib, "binding_present", lambda: False)
    elif not _lib.binding_present():
        pytest.skip("the torch binding is not built")


LAYERS = {"linear": lambda: nn.Linear(4, 4), "linear_no_bias": lambda: nn.Linear(4, 4, bias=False),
          "conv1d": lambda: Conv1D(4, 4)}
SHAPES = {"2d": (3, 4), "3d": (3, 2, 4)}


class Hooked:
    """A layer with the pair on it; ``seen`` collects the (input, gradient) that the hook was given."""

    def __init__(self, kind, shape):
        torch.manual_seed(0)
        self.layer, self.seen = LAYERS[kind](), []
        self.x = torch.randn(SHAPES[shape], requires_grad=True) * 1
        self.handles = register_hook_pair(self.layer, self.capture, self.hook, "kept")

    @staticmethod
    def capture(layer, inputs, outputs):
        if torch.is_grad_enabled():
            layer.__dict__["kept"] = inputs[0].detach()

    def hook(self, layer, grad_input, grad_output):
        A = layer.__dict__.pop("kept", None)
        if A is None:
            raise RuntimeError("no input kept")
        self.seen.append((A, grad_output[0].clone()))

    def check(self, calls=1):
        """The hook's products add up to autograd's weight gradient."""
        assert len(self.seen) == calls
        total = sum(A.reshape(-1, 4).t() @ g.reshape(-1, 4) for A, g in self.seen)
        want = self.layer.weight.grad
        torch.testing.assert_close(total, want if isinstance(self.layer, Conv1D) else want.t(), rtol=1e-5, atol=1e-5)


every_layer = pytest.mark.parametrize("kind", LAYERS)
every_shape = pytest.mark.parametrize("shape", SHAPES)


@every_layer
@every_shape
def test_a_users_tensor_hook_comes_first(kind, shape):
    h = Hooked(kind, shape)
    y = h.layer(h.x)
    y.register_hook(lambda g: g * 10)
    (y ** 2).sum().backward()
    h.check()


@every_layer
@every_shape
def test_a_users_module_hooks(kind, shape):
    h = Hooked(kind, shape)
    order = []
    h.layer.register_full_backward_pre_hook(lambda m, g: (g[0] * 3,))
    h.layer.register_full_backward_hook(lambda m, gi, go: order.append(len(h.seen)))
    (h.layer(h.x) ** 2).sum().backward()
    h.check()
    assert order == [1]                  # after this pair's hook, whose results it may read


@every_layer
@every_shape
def test_gradients_up_to_the_output_call_nothing(kind, shape):
    h = Hooked(kind, shape)
    y = h.layer(h.x)
    loss = (y ** 2).sum()
    torch.autograd.grad(loss, y, retain_graph=True)
    assert not h.seen
    loss.backward()
    h.check()


@every_layer
@every_shape
@pytest.mark.parametrize("when", ["none", "before", "after"])
def test_in_place_operation_on_the_output(kind, shape, when):
    h = Hooked(kind, shape)
    y = h.layer(h.x)
    if when == "before":
        y.register_hook(lambda g: g * 10)
    z = F.relu(y, inplace=True)
    if when == "after":
        z.register_hook(lambda g: g * 10)
    (z ** 2).sum().backward()
    h.check()


def test_output_that_is_part_of_its_base():
    """A view whose elements are not its base's in order: the hook stays at the view's own node."""
    class Turned(nn.Linear):
        def forward(self, x):
            return super().forward(x).transpose(0, 1)

    LAYERS["turned"] = lambda: Turned(4, 4)
    try:
        h = Hooked("turned", "3d")
    finally:
        del LAYERS["turned"]
    (h.layer(h.x) ** 2).sum().backward()
    (A, g), = h.seen
    assert g.shape == (2, 3, 4)
    torch.testing.assert_close(A.reshape(-1, 4).t() @ g.transpose(0, 1).reshape(-1, 4), h.layer.weight.grad.t())


@every_layer
@every_shape
@pytest.mark.parametrize("reentrant", [False, True])
def test_shared_layer_under_checkpointing(kind, shape, reentrant):
    """Both calls are consumed, each with its own input, and nothing stays behind."""
    h = Hooked(kind, shape)
    x = h.x
    for _ in range(2):
        x = checkpoint(lambda t: h.layer(t).relu(), x, use_reentrant=reentrant)
    (x ** 2).sum().backward()
    h.check(calls=2)
    assert not any(a.startswith("kept") for a in h.layer.__dict__)


@every_layer
@every_shape
def test_shared_layer_with_one_call_checkpointed(kind, shape):
    h = Hooked(kind, shape)
    x = checkpoint(lambda t: h.layer(t).relu(), h.x, use_reentrant=False)
    (h.layer(x) ** 2).sum().backward()
    h.check(calls=2)


@every_layer
@every_shape
@pytest.mark.parametrize("block", ["ends in the layer", "goes on"])
def test_checkpointed_block(kind, shape, block):
    h = Hooked(kind, shape)
    tail = (lambda t: t) if block == "ends in the layer" else (lambda t: (t ** 2).sin())
    x = checkpoint(lambda t: tail(h.layer(t.relu() * 2)), h.x, use_reentrant=False)
    (x ** 2).sum().backward()
    h.check()
    assert not any(a.startswith("kept") for a in h.layer.__dict__)


@every_layer
@every_shape
def test_shared_layer_without_recomputation_is_refused(kind, shape):
    h = Hooked(kind, shape)
    with pytest.raises(RuntimeError, match="no input kept"):
        h.layer(h.layer(h.x).relu()).sum().backward()


@every_layer
@every_shape
def test_another_forward_before_the_backward_pass(kind, shape):
    """The hook gets the input of the call that is differentiated, not the last one's."""
    h = Hooked(kind, shape)
    loss = (h.layer(h.x) ** 2).sum()
    h.layer(h.x * 5 + 1)
    loss.backward()
    h.check()


def test_two_pairs_on_one_layer():
    h = Hooked("linear", "3d")
    other = []
    register_hook_pair(h.layer, lambda m, i, o: m.__dict__.__setitem__("second", i[0].detach()),
                       lambda m, gi, go: other.append(m.__dict__.pop("second")), "second")
    (h.layer(h.x) ** 2).sum().backward()
    h.check()
    assert torch.equal(other[0], h.x)


def test_layer_that_returns_its_parameter():
    class Table(nn.Linear):
        def forward(self, x):
            return self.weight

    LAYERS["table"] = lambda: Table(4, 4)
    try:
        h = Hooked("table", "2d")
    finally:
        del LAYERS["table"]
    (h.layer(h.x) * 3).sum().backward()
    (A, g), = h.seen
    assert torch.equal(A, h.x) and torch.equal(g, torch.full((4, 4), 3.0))


@every_layer
def test_tracing_a_hooked_layer_is_refused(kind):
    h = Hooked(kind, "3d")
    with pytest.raises(ValueError, match="backward hooks"):
        torch.jit.trace(nn.Sequential(h.layer), (h.x.detach(),))
    (h.layer(h.x) ** 2).sum().backward()          # and it goes on as before
    h.check()
    for handle in h.handles:
        handle.remove()
    torch.jit.trace(nn.Sequential(h.layer), (h.x.detach(),))


def test_exceptions_of_the_hook_reach_the_caller():
    layer = nn.Linear(4, 4)

    def fail(m, grad_input, grad_output):
        raise KeyError("from the hook")

    register_hook_pair(layer, Hooked.capture, fail, "kept")
    with pytest.raises(KeyError, match="from the hook"):
        layer(torch.randn(3, 4, requires_grad=True)).sum().backward()


def test_compiled_model():
    h = Hooked("linear", "3d")
    torch._dynamo.reset()
    (torch.compile(nn.Sequential(h.layer, nn.Tanh()), backend="eager")(h.x) ** 2).sum().backward()
    h.check()


@pytest.mark.parametrize("backward", [False, True])
def test_a_layer_that_holds_its_output_is_collected(backward):
    """The hook sits in the graph, the graph on the output, the output on the layer."""
    seen = []
    layer = nn.Linear(4, 4)
    register_hook_pair(layer, Hooked.capture, lambda m, grad_input, grad: seen.append(m.__dict__.pop("kept").shape), "kept")
    layer.seen_output = layer(torch.randn(3, 2, 4))
    if backward:
        layer.seen_output.sum().backward()
        assert seen == [(3, 2, 4)]
    gone = weakref.ref(layer)
    del layer
    gc.collect()
    assert gone() is None


def test_a_graph_that_outlives_its_backward_pass_keeps_no_input():
    h = Hooked("linear", "3d")
    loss = (h.layer(h.x * 2) ** 2).sum()
    kept = weakref.ref(h.layer.__dict__["kept"])
    loss.backward()
    h.seen.clear()
    gc.collect()
    assert kept() is None and loss.grad_fn is not None
