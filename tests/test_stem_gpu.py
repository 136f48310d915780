"""The stem's staged path (in-plane neighbourhoods) against fp64, exact: operands are -1 / 0 / 1."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _tri(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-1, 2, shape, generator=g, device="cuda").float()


@pytest.mark.parametrize("dims,cin,cout,dtype,bias", [
    ((1, 1, 8, 16), 3, 64, torch.float32, False), ((2, 5, 9, 17), 3, 64, torch.float32, False),
    ((1, 4, 16, 32), 3, 32, torch.bfloat16, True), ((1, 7, 23, 41), 2, 16, torch.float32, True),
    ((3, 2, 10, 19), 1, 128, torch.float32, False), ((1, 3, 8, 100), 3, 24, torch.float32, True),
    ((1, 33, 40, 48), 3, 48, torch.float32, False), ((1, 20, 12, 24), 3, 192, torch.bfloat16, False)])
def test_stem_forward_and_weight_gradient(dims, cin, cout, dtype, bias, monkeypatch):
    from scaffold_b200.ops import _lib, conv3d
    n, d, h, w = dims
    x, wt, gy = _tri((n, cin, d, h, w), 1), _tri((cout, cin, 3, 3, 3), 2), _tri((n, cout, d, h, w), 3)
    b = _tri((cout,), 4)
    conv = conv3d.Conv3d(cin, cout, 3, padding=1, bias=bias).cuda()
    with torch.no_grad():
        conv.weight.copy_(wt)
        if bias:
            conv.bias.copy_(b)
    calls = []
    real = conv3d.ck.stage_stem
    monkeypatch.setattr(conv3d.ck, "stage_stem", lambda t: calls.append(1) or real(t))
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = conv(x.to(dtype))
    y.backward(gy.to(y.dtype))
    torch.cuda.synchronize()
    _lib.check_status()
    assert calls
    ref = F.conv3d(x.double(), wt.double(), b.double() if bias else None, padding=1).round()
    assert torch.equal(y.double(), ref.to(torch.bfloat16).double())
    gw = torch.nn.grad.conv3d_weight(x.double(), wt.shape, gy.double(), padding=1).round()
    assert torch.equal(conv.weight.grad.double(), gw)  # integers below 2^24: exact in fp32
    if bias:
        assert torch.equal(conv.bias.grad.double(), gy.double().sum((0, 2, 3, 4)))


@pytest.mark.parametrize("dims,cout", [((2, 6, 20, 24), 64), ((1, 9, 8, 16), 32)])
def test_stem_statistics_describe_its_output(dims, cout):
    from scaffold_b200.ops import conv3d, gn_kernels as gk
    n, d, h, w = dims
    conv = conv3d.Conv3d(3, cout, 3, padding=1, bias=False).cuda()
    conv.gn_groups_hint = 8
    with torch.autocast("cuda", dtype=torch.bfloat16), torch.no_grad():
        y = conv(torch.rand((n, 3, d, h, w), device="cuda"))
    part, splits, groups = y._sb_gn_partials
    fin = gk.gn_finalize(part, n, groups, splits).view(n, groups, 3).double()
    v = y.double().reshape(n, groups, -1)
    assert torch.equal(fin[..., 0], torch.full_like(fin[..., 0], v.shape[2]))
    # fp32 sums of at most 128 x 8 values per partial, then fp64: errors of a few 2^-24 of the largest terms
    torch.testing.assert_close(fin[..., 1], v.mean(2), rtol=0, atol=2e-6 * float(v.abs().max()))
    torch.testing.assert_close(fin[..., 2] / v.shape[2], v.var(2, unbiased=False), rtol=1e-5, atol=0)
