"""When a backward pass may add a parameter's gradient to the flat buffer itself (host logic, on a stand-in layer)."""
import pytest
import torch

from scaffold_b200.ops import layout


class _Scale(torch.autograd.Function):
    """y = w * x with the rule of the kernels' layers."""

    @staticmethod
    def forward(ctx, w, x):
        ctx.wparam, ctx.x = w, x
        return w * x

    @staticmethod
    def backward(ctx, g):
        direct = layout.direct_grad_target(ctx.wparam, ctx)
        if direct is None:
            return g * ctx.x, g * ctx.wparam
        with torch.no_grad():
            direct.add_(g * ctx.x)
        layout.notify_grad_written(ctx.wparam)
        return None, g * ctx.wparam


@pytest.fixture
def param():
    w = torch.nn.Parameter(torch.tensor([1.0, 2.0, 3.0]))
    w.grad = torch.zeros(3)
    setattr(w, layout.FLAT_GRAD_ATTR, True)
    told = []

    def listener(p):
        told.append(p)
    before = list(layout._grad_written_listeners)
    layout.add_grad_written_listener(listener)
    w.told = told
    yield w
    layout._grad_written_listeners[:] = before


X = torch.tensor([5.0, 6.0, 7.0])


def test_backward_writes_directly(param):
    buffer = param.grad
    for k in (1, 2):
        _Scale.apply(param, X).sum().backward()
        assert param.grad is buffer and torch.equal(buffer, k * X) and len(param.told) == k
    _Scale.apply(param, X).sum().backward(inputs=[param])
    assert torch.equal(buffer, 3 * X) and len(param.told) == 3


def test_autograd_grad_returns_the_gradient_and_leaves_the_buffer(param):
    (g,) = torch.autograd.grad(_Scale.apply(param, X).sum(), [param])
    assert torch.equal(g, X) and not param.grad.any() and not param.told


def test_gradients_of_other_tensors_leave_the_buffer(param):
    x = X.clone().requires_grad_()
    (g,) = torch.autograd.grad(_Scale.apply(param, x).sum(), [x])
    _Scale.apply(param, x).sum().backward(inputs=[x])
    assert torch.equal(g, param.detach()) and torch.equal(x.grad, param.detach())
    assert not param.grad.any() and not param.told


def test_hooks_of_the_caller_fire(param):
    """A post-accumulate hook runs after the direct write too: autograd calls it although it added nothing itself."""
    seen = []
    handle = param.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
    _Scale.apply(param, X).sum().backward()
    assert len(seen) == 1 and torch.equal(seen[0], X) and len(param.told) == 1
    handle.remove()
    handle = param.register_hook(lambda g: seen.append(g))
    _Scale.apply(param, X).sum().backward()
    assert len(seen) == 2 and torch.equal(seen[1], X) and len(param.told) == 1
    handle.remove()
