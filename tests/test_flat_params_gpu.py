"""Parameters of a flat optimizer: gradients written straight into the flat buffer, operand copies per optimizer (GPU)."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(seed, c=32):
    from scaffold_b200.ops.conv3d import Conv3d, ConvTranspose3d
    from scaffold_b200.ops.group_norm import GroupNorm
    torch.manual_seed(seed)
    return torch.nn.Sequential(ConvTranspose3d(c, c, 2, 2), Conv3d(c, 64, 3, padding=1, bias=False),
                               GroupNorm(8, 64, activation="relu"), Conv3d(64, 16, 1)).cuda()


def _run(net, x):
    with torch.autocast("cuda", dtype=torch.bfloat16):
        return net(x)


@pytest.mark.parametrize("n,edge", [(1, (4, 4, 8)), (3, (5, 6, 9))])
def test_direct_gradients_accumulate_like_autograd(n, edge):
    from scaffold_b200.ops.optim import FusedClipAdam
    plain = _net(0)
    flat = copy.deepcopy(plain)
    FusedClipAdam(flat.parameters()).attach()
    x = torch.randn((n, 32, *edge), device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last_3d)
    seen, added = [], []
    handle = flat[2].weight.register_hook(lambda g: seen.append(g.clone()))
    for p in (flat[2].bias, flat[3].bias, flat[1].weight):
        p.register_post_accumulate_grad_hook(lambda p: added.append(p))
    for k in range(2):  # the second pass adds to the first: twice the gradient, exactly
        for net in (plain, flat):
            _run(net, x).float().square().mean().backward()
        if k == 0:
            handle.remove()
    assert len(added) == 6  # a post-accumulate hook runs after a direct write as well
    assert len(seen) == 1 and seen[0].shape == flat[2].weight.shape  # a hooked parameter keeps autograd's path
    for (name, p), q in zip(plain.named_parameters(), flat.parameters()):
        # the same kernels in the same order; only the reduction that adds into an existing value may round once more
        torch.testing.assert_close(q.grad, p.grad, rtol=2 ** -22, atol=0, msg=name)


@pytest.mark.parametrize("name", ["0.weight", "0.bias", "1.weight", "2.weight", "2.bias", "3.weight", "3.bias"])
def test_gradients_asked_for_by_name_are_returned(name):
    """autograd.grad() of a flat optimizer's parameter, and backward(inputs=...) without it, leave its .grad alone."""
    from scaffold_b200.ops.optim import FusedClipAdam
    plain = _net(0)
    flat = copy.deepcopy(plain)
    FusedClipAdam(flat.parameters()).attach()
    x = torch.randn((2, 32, 4, 6, 8), device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last_3d)
    loss = lambda net, t: _run(net, t).float().square().mean()  # noqa: E731
    want, got = (torch.autograd.grad(loss(net, x), [dict(net.named_parameters())[name]])[0] for net in (plain, flat))
    assert torch.equal(got, want)
    x.requires_grad_()
    loss(flat, x).backward(inputs=[x])
    assert x.grad.any() and all(not p.grad.any() for p in flat.parameters())


def test_a_step_renews_its_own_operand_copies_only():
    from scaffold_b200.ops import _lib
    from scaffold_b200.ops.optim import FusedClipAdam
    nets = [_net(1), _net(2)]
    opts = [FusedClipAdam(n.parameters(), lr=1e-2) for n in nets]
    for o in opts:
        o.attach()
    x = torch.randn((1, 32, 4, 8, 8), device="cuda").to(torch.bfloat16)
    for net, o in zip(nets, opts):
        _run(net, x).float().square().mean().backward()
        o.step()
    with torch.no_grad():
        other = _run(nets[1], x).clone()
        before = _lib.launch_count()
        again = _run(nets[1], x)
        steady = _lib.launch_count() - before
        opts[0].step()
        before = _lib.launch_count()
        after = _run(nets[1], x)
        assert _lib.launch_count() - before == steady  # nothing of the second network was packed anew
        assert torch.equal(other, again) and torch.equal(other, after)
        got = _run(nets[0], x)
        fresh = _net(9)
        fresh.load_state_dict(nets[0].state_dict())
        assert torch.equal(got, _run(fresh, x))        # the first network runs on its new weights
        nets[0][1].weight.mul_(2.0)                    # and follows a change that no optimizer made
        fresh[1].weight.mul_(2.0)
        assert torch.equal(_run(nets[0], x), _run(fresh, x))
