"""Pooling that adds the skip connection's gradient in its backward pass: the bits of the two separate passes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 2, 2, 2, 8), (2, 4, 6, 10, 32), (1, 3, 5, 7, 16), (2, 9, 4, 11, 64), (1, 16, 16, 17, 24)])
def test_sum_of_both_gradients(shape):
    from scaffold_b200.ops import pool_kernels as pk
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    n, d, h, w, c = shape
    gy = torch.randn((n, d // 2, h // 2, w // 2, c), generator=g, device="cuda").to(torch.bfloat16)
    gs = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    y, idx = pk.maxpool2_fwd_idx(x)
    want = pk.maxpool2_bwd_idx(gy, idx, shape) + gs
    for use_pool, use_skip, expect in ((True, True, want), (True, False, pk.maxpool2_bwd_idx(gy, idx, shape)),
                                       (False, True, gs)):
        xl = x.clone().requires_grad_(True)
        pooled, skip = pk.MaxPool2SkipFn.apply(xl)
        assert torch.equal(pooled, y) and torch.equal(skip, x)
        outs = [t for t, use in ((pooled, use_pool), (skip, use_skip)) if use]
        torch.autograd.backward(outs, [t for t, use in ((gy, use_pool), (gs, use_skip)) if use])
        assert torch.equal(xl.grad, expect)


@pytest.mark.parametrize("dims", [(16, 16, 32), (18, 20, 22)])
@pytest.mark.parametrize("where", ["block", "sequence", "pool"])
def test_a_hook_on_a_passed_by_module_keeps_its_call(dims, where):
    from scaffold_b200.models.unet import UNet
    torch.manual_seed(0)
    net = UNet(3, 4, layers=2, base_width=16).cuda()
    x = torch.rand((1, 3, *dims), device="cuda")

    def grads():
        net.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            net(x).float().square().mean().backward()
        return [p.grad.clone() for p in net.parameters()]

    fused = grads()
    block = net.down_list[1]
    seen = []
    mod = {"block": block, "sequence": block.maxpool_conv, "pool": block.maxpool_conv[0]}[where]
    handle = mod.register_forward_hook(lambda *a: seen.append(1))
    separate = grads()
    handle.remove()
    assert seen
    for a, b in zip(fused, separate):
        assert torch.equal(a, b)


@pytest.mark.parametrize("where", ["block", "double", "sequence", "convolution"])
def test_a_hook_that_changes_the_skip_tensor_may_do_so(where):
    """In place, as on any module's input; and the gradient that it waits for is the whole one."""
    from scaffold_b200.models.unet import UNet
    torch.manual_seed(0)
    net = UNet(3, 4, layers=2, base_width=16).cuda()
    x = torch.rand((1, 3, 16, 16, 32), device="cuda")
    up = net.up_list[1]   # reads the first block's output
    mod = {"block": up, "double": up.conv, "sequence": up.conv.double_conv, "convolution": up.conv.double_conv[0]}[where]
    whole, inside = [], []

    def outer(m, args, out):
        out.register_hook(lambda g: whole.append(g.clone()))

    def inner(m, args):
        skip = args[1] if where == "block" else args[0][0]
        skip.register_hook(lambda g: inside.append(g.clone()))
        with torch.no_grad():
            skip.mul_(0.5)
        return None
    handles = [net.down_list[0].register_forward_hook(outer), mod.register_forward_pre_hook(inner)]
    with torch.autocast("cuda", dtype=torch.bfloat16):
        net(x).float().square().mean().backward()
    for h in handles:
        h.remove()
    assert len(whole) == len(inside) == 1 and torch.equal(whole[0], inside[0])


def test_a_run_of_its_own_is_called_for_every_block():
    from scaffold_b200.models.unet import UNet

    class Counting(UNet):
        calls = 0

        def _run(self, block, *inputs):
            self.calls += 1
            return super()._run(block, *inputs)
    net = Counting(3, 4, layers=2, base_width=16).cuda()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        net(torch.rand((1, 3, 16, 16, 32), device="cuda")).sum().backward()
    assert net.calls == 3 + 3   # three encoder blocks, two decoder blocks, the head
