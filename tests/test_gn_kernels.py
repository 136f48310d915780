"""GPU parity of the channels-last GroupNorm(+ReLU) kernels against float64 PyTorch."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, G, D, H, W, relu
    (2, 64, 8, 8, 16, 16, True),
    (1, 128, 8, 4, 8, 8, True),
    (2, 16, 8, 4, 8, 8, True),
    (1, 32, 8, 5, 7, 9, False),
    (1, 1024, 8, 2, 4, 4, True),
    (1, 64, 8, 32, 32, 32, True),
]


def _ref(x, w, b, G, relu):
    y = F.group_norm(x, G, w, b, 1e-5)
    return F.relu(y) if relu else y


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_gn_forward_backward(case):
    from scaffold_b200.ops import gn_kernels as gk
    n, c, G, d, h, w, relu = case
    g = torch.Generator(device="cuda").manual_seed(0)
    x = (torch.randn((n, c, d, h, w), generator=g, device="cuda") * 2 + 3).to(torch.bfloat16)
    wt = torch.randn(c, generator=g, device="cuda")
    bs = torch.randn(c, generator=g, device="cuda")
    dy = torch.randn((n, c, d, h, w), generator=g, device="cuda").to(torch.bfloat16)
    xv = x.permute(0, 2, 3, 4, 1).contiguous()
    dyv = dy.permute(0, 2, 3, 4, 1).contiguous()
    y, mean, rstd = gk.gn_forward(xv, wt, bs, G, 1e-5, relu)
    xd = x.double().requires_grad_(True)
    wd = wt.double().requires_grad_(True)
    bd = bs.double().requires_grad_(True)
    ref = _ref(xd, wd, bd, G, relu)
    got = y.permute(0, 4, 1, 2, 3).double()
    # bf16 output: half an ulp of the reference magnitude
    tol = ref.detach().abs().clamp_min(1.0) * 2 ** -8
    assert ((got - ref.detach()).abs() <= tol).all()
    xg = xd.detach().reshape(n, G, -1)
    assert torch.allclose(mean.double(), xg.mean(-1), atol=1e-4, rtol=1e-5)
    assert torch.allclose(rstd.double(), (xg.var(-1, unbiased=False) + 1e-5).rsqrt(), atol=1e-4, rtol=1e-4)
    ref.backward(dy.double())
    dx, dw, db = gk.gn_backward(dyv, xv, wt, bs, mean, rstd, G, 1e-5, relu)
    gdx = dx.permute(0, 4, 1, 2, 3).double()
    scale = xd.grad.abs().max().item()
    assert (gdx - xd.grad).abs().max().item() <= scale * 2 ** -7 + 1e-6
    assert torch.allclose(dw.double(), wd.grad, rtol=2e-3, atol=2e-3 * wd.grad.abs().max().item())
    assert torch.allclose(db.double(), bd.grad, rtol=2e-3, atol=2e-3 * bd.grad.abs().max().item())


def test_gn_large_mean_is_stable():
    """Shifted/Welford statistics: a large common offset must not destroy the variance."""
    from scaffold_b200.ops import gn_kernels as gk
    g = torch.Generator(device="cuda").manual_seed(1)
    x = (torch.randn((1, 64, 8, 16, 16), generator=g, device="cuda") + 200.0).to(torch.bfloat16)
    w = torch.ones(64, device="cuda")
    b = torch.zeros(64, device="cuda")
    xv = x.permute(0, 2, 3, 4, 1).contiguous()
    _, mean, rstd = gk.gn_forward(xv, w, b, 8, 1e-5, False)
    xg = x.double().reshape(1, 8, -1)
    assert torch.allclose(mean.double(), xg.mean(-1), rtol=1e-6)
    assert torch.allclose(rstd.double(), (xg.var(-1, unbiased=False) + 1e-5).rsqrt(), rtol=1e-3)


def test_gn_two_shards_equal_whole_volume():
    """Merging a neighbour's partials reproduces the unsharded statistics (emulated on one GPU)."""
    from scaffold_b200.ops import gn_kernels as gk
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((1, 8, 16, 16, 64), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(64, generator=g, device="cuda")
    b = torch.randn(64, generator=g, device="cuda")
    whole, mean, rstd = gk.gn_forward(x, w, b, 8)
    halves = [x[:, :4].contiguous(), x[:, 4:].contiguous()]
    parts = [gk.gn_stats(hv, w, b, 8, 1e-5, True) for hv in halves]
    outs = []
    for i, hv in enumerate(halves):
        order = [parts[i].data_ptr(), parts[1 - i].data_ptr()]
        y, m, r = gk.gn_apply(hv, w, b, 8, 1e-5, True, order, shards=2)
        outs.append(y)
        assert torch.allclose(m, mean, rtol=1e-5, atol=1e-6)
        assert torch.allclose(r, rstd, rtol=1e-5)
    got = torch.cat(outs, 1).float()
    assert (got - whole.float()).abs().max().item() <= 2 ** -6


@pytest.mark.parametrize("shape,groups", [((2, 16, 32, 32, 64), 8), ((1, 8, 8, 8, 1024), 8), ((3, 5, 9, 7, 32), 4),
                                          ((1, 8, 8, 16, 64), 8), ((1, 1, 24, 44, 64), 8), ((4, 8, 16, 16, 256), 8),
                                          ((1, 32, 32, 32, 64), 8)])
def test_last_block_collapse_equals_the_separate_finalize_launch(shape, groups, monkeypatch):
    """The statistics kernels can collapse their partials in the block that finishes last; the result must be the
    bits of the separate finalize launch (same order of the sums), forward and backward. The shapes have 5 to 592
    partials per output, 32 and 33 (one warp, four warps) among them."""
    from scaffold_b200.ops import _lib, gn_kernels as gk
    g = torch.Generator(device="cuda").manual_seed(21)
    x = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    c = shape[-1]
    w = torch.rand(c, generator=g, device="cuda") + 0.5
    b = torch.randn(c, generator=g, device="cuda")
    outs = []
    for fused in (True, False):
        monkeypatch.setattr(gk, "_FUSED_FINALIZE", fused)
        fin = gk.gn_stats(x, w, b, groups, 1e-5, True)
        _, mean, rstd = gk.gn_apply(x, w, b, groups, 1e-5, True, [fin.data_ptr()])
        # backward sums: the fused form is used only for a handful of outputs, so ask for it directly as well
        a = gk._base(x, w, b, groups, 1e-5, True, 1)
        a.dy, a.mean, a.rstd = dy.data_ptr(), mean.data_ptr(), rstd.data_ptr()
        part = torch.empty(gk.partial_numel_bwd(x), dtype=torch.float32, device="cuda")
        bfin = torch.empty(shape[0] * c * 2, dtype=torch.float32, device="cuda")
        a.part = part.data_ptr()
        a.n_parts = 1
        a.parts[0] = part.data_ptr()
        if fused:
            a.fin = bfin.data_ptr()
        _lib.check(_lib.lib().sb_gn_bwd_partial(C.byref(a), _lib.stream_ptr()), "sb_gn_bwd_partial")
        if not fused:
            _lib.check(_lib.lib().sb_gn_bwd_finalize(part.data_ptr(), bfin.data_ptr(), shape[0], c, a.nsplit,
                                                     _lib.stream_ptr()), "sb_gn_bwd_finalize")
        torch.cuda.synchronize()
        outs.append((fin.clone(), bfin.clone()))
    assert torch.equal(outs[0][0], outs[1][0])
    assert torch.equal(outs[0][1], outs[1][1])
    # a second fused launch finds its ticket counter back at zero
    monkeypatch.setattr(gk, "_FUSED_FINALIZE", True)
    again = gk.gn_stats(x, w, b, groups, 1e-5, True)
    torch.cuda.synchronize()
    assert torch.equal(again, outs[0][0])


@pytest.mark.parametrize("nsplit", [1, 31, 32, 33, 128, 129, 592, 1024, 1025, 2049, 16384])
def test_finalize_pools_partials_like_fp64(nsplit):
    """All three collapse kernels (a warp per output up to 32 partials, a block up to 1024, a cluster of eight CTAs
    beyond), empty partials and a mean of a hundred standard deviations included."""
    from scaffold_b200.ops import gn_kernels as gk
    g = torch.Generator(device="cuda").manual_seed(nsplit)
    part = torch.empty((2, nsplit, 8, 3), device="cuda")
    part[..., 0] = torch.randint(0, 3, (2, nsplit, 1), generator=g, device="cuda") * 512.0
    part[:, 0, :, 0] = 512.0
    part[..., 1] = 100.0 + torch.randn((2, nsplit, 8), generator=g, device="cuda")
    part[..., 2] = torch.rand((2, nsplit, 8), generator=g, device="cuda") * 512.0
    got = gk.gn_finalize(part.reshape(-1), 2, 8, nsplit).view(2, 8, 3).double()
    n, m, m2 = part.double().unbind(-1)
    tot = n.sum(1)
    mean = (n * m).sum(1) / tot
    ref = torch.stack([tot, mean, (m2 + n * (m - mean[:, None]) ** 2).sum(1)], -1)
    # sums in double, results rounded once to fp32: 2^-24, doubled for the subtraction in M2
    torch.testing.assert_close(got, ref, rtol=2 ** -22, atol=1e-3)


@pytest.mark.parametrize("nsplit", [1, 32, 33, 1024, 1025])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_finalize_keeps_what_is_not_finite(nsplit, bad):
    """A partial over an infinity has that mean and a NaN for M2; its group's variance is NaN, as the formula's is."""
    from scaffold_b200.ops import gn_kernels as gk
    part = torch.ones((2, nsplit, 8, 3), device="cuda")
    part[1, nsplit // 2, 3, 1], part[1, nsplit // 2, 3, 2] = bad, float("nan")
    got = gk.gn_finalize(part.reshape(-1), 2, 8, nsplit).view(2, 8, 3)
    expect = torch.zeros((2, 8), dtype=torch.bool, device="cuda")
    expect[1, 3] = True
    assert torch.equal(got[..., 2].isnan(), expect) and torch.equal(~got[..., 1].isfinite(), expect)


@pytest.mark.parametrize("dims", [(4, 5, 6), (24, 24, 24)])
@pytest.mark.parametrize("through", ["statistics", "convolution"])
def test_an_infinite_activation_makes_its_group_nan(dims, through):
    from scaffold_b200.ops.conv3d import Conv3d
    from scaffold_b200.ops.group_norm import GroupNorm
    torch.manual_seed(0)
    x = torch.randn((2, 64, *dims), device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last_3d)
    norm = GroupNorm(8, 64, activation="relu").cuda()
    conv = Conv3d(64, 64, 3, padding=1, bias=False).cuda()
    conv.gn_groups_hint = 8
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        if through == "convolution":
            conv.weight[17] = 3e38   # its output overflows where the inputs add up
            x[1] = x[1].abs() * 100
            x[0] = 0
            y = norm(conv(x))
        else:
            x[1, 17, 1, 2, 3] = float("inf")
            y = norm(x)
    assert y[1, 16:24].isnan().all() and not y[0].isnan().any()
    assert not y[1, :16].isnan().any() and not y[1, 24:].isnan().any()
