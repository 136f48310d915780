"""The generic convolution kernel's store paths and split reduction at ragged sizes, exact against fp64.

Operands are -1 / 0 / 1, so every sum is an integer below 2^24: fp32 accumulation is exact in any order and the bf16
result must be the rounded fp64 one.
"""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _tri(shape, seed, density=0.5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(shape, generator=g, device="cuda")
    return (u > 1 - density / 2).float() - (u < density / 2).float()


def _vm(x):
    return x.permute(0, 2, 3, 4, 1).to(torch.bfloat16).contiguous()


def _nc(y):
    return y.permute(0, 4, 1, 2, 3).double()


def _bf(x):
    return x.round().to(torch.bfloat16).double()


@pytest.mark.parametrize("dims,cin,cout", [
    ((1, 1, 1, 1), 16, 16), ((1, 3, 5, 7), 64, 32), ((2, 5, 9, 13), 32, 48), ((1, 2, 8, 8), 16, 64),
    ((1, 7, 11, 23), 16, 128), ((3, 4, 6, 31), 128, 256), ((1, 1, 1, 129), 64, 9)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_pointwise(dims, cin, cout, with_bias):
    from scaffold_b200.ops import _lib, conv_kernels as ck
    n, d, h, w = dims
    x, wt = _tri((n, cin, d, h, w), 1), _tri((cout, cin, 1, 1, 1), 2)
    bias = _tri((cout,), 3) if with_bias else None
    cpad = ck.pad_channels(cout)
    bpad = F.pad(bias, (0, cpad - cout)) if with_bias else None
    (y,) = ck.conv_same([_vm(x)], ck.pack_weight_fwd(wt), 1, [cpad], bias=bpad)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = F.conv3d(x.double(), wt.double(), None if bias is None else bias.double())
    assert torch.equal(_nc(y)[:, :cout], _bf(ref))


@pytest.mark.parametrize("dims,cin,cout", [
    ((1, 1, 1, 1), 32, 16), ((1, 3, 5, 7), 64, 32), ((2, 5, 3, 9), 96, 48), ((1, 2, 9, 17), 128, 64),
    ((2, 3, 4, 33), 32, 16), ((1, 2, 3, 5), 16, 8), ((1, 2, 2, 150), 256, 128), ((1, 1, 2, 3), 16, 6144),
    ((1, 1, 2, 3), 16, 20000)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_transposed(dims, cin, cout, with_bias):
    from scaffold_b200.ops import _lib, conv_kernels as ck
    n, d, h, w = dims
    x, wt = _tri((n, cin, d, h, w), 4), _tri((cin, cout, 2, 2, 2), 5)
    bias = _tri((cout,), 6) if with_bias else None
    y = ck.convT_fwd(_vm(x), ck.pack_weight_convT_fwd(wt), cout, bias)
    gy = _tri((n, cout, 2 * d, 2 * h, 2 * w), 7)
    gx = ck.convT_dgrad(_vm(gy), ck.pack_weight_convT_dgrad(wt), cin)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = F.conv_transpose3d(x.double(), wt.double(), None if bias is None else bias.double(), stride=2)
    assert torch.equal(_nc(y), _bf(ref))
    assert torch.equal(_nc(gx), _bf(F.conv3d(gy.double(), wt.double(), stride=2)))


@pytest.mark.parametrize("dims,cins,couts", [
    ((1, 5, 7, 9), [512], [128]), ((1, 6, 5, 7), [256, 256], [256]), ((2, 3, 7, 15), [64], [64, 64]),
    ((1, 4, 4, 4), [128], [32, 32]), ((1, 11, 6, 9), [128], [16, 48]), ((1, 1, 1, 1), [128], [64]),
    ((1, 20, 7, 40), [128], [128]), ((1, 12, 20, 12), [32], [64]), ((1, 2, 3, 4), [48], [16])])
def test_small_volumes_split_and_whole_reductions(dims, cins, couts):
    from scaffold_b200.ops import _lib, conv_kernels as ck
    n, d, h, w = dims
    xs = [_tri((n, c, d, h, w), 8 + i) for i, c in enumerate(cins)]
    wt = _tri((sum(couts), sum(cins), 3, 3, 3), 10)
    ys = ck.conv_same([_vm(x) for x in xs], ck.pack_weight_fwd(wt), 3, couts)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = F.conv3d(torch.cat(xs, 1).double(), wt.double(), padding=1)
    assert torch.equal(torch.cat([_nc(y) for y in ys], 1), _bf(ref))


@pytest.mark.parametrize("voxels", [1, 7, 8, 9, 16, 17, 129, 5000, 150001])
@pytest.mark.parametrize("cin,cout", [(16, 64), (32, 64), (16, 32), (16, 16), (32, 48), (32, 128)])
def test_few_channels_pointwise(voxels, cin, cout):
    """Fragments of 16 voxels, a ragged last one; without a bias (the head's backward-data)."""
    from scaffold_b200.ops import _lib, conv_kernels as ck
    x, wt = _tri((1, cin, 1, 1, voxels), 11), _tri((cout, cin, 1, 1, 1), 12)
    out = torch.full((1, 1, 1, voxels + 1, cout), 7.0, dtype=torch.bfloat16, device="cuda")  # one voxel more than is written
    ck.conv_same([_vm(x)], ck.pack_weight_fwd(wt), 1, [cout], out=[out[:, :, :, :voxels]])
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(_nc(out[:, :, :, :voxels]), _bf(F.conv3d(x.double(), wt.double())))
    assert bool((out[:, :, :, voxels] == 7).all())


@pytest.mark.parametrize("cin,cout", [(16, 8), (32, 16), (48, 40), (64, 32), (96, 72), (128, 64)])
def test_packed_operands_equal_the_general_packing(cin, cout):
    from scaffold_b200.ops import conv_kernels as ck
    wt = torch.randn((cin, cout, 2, 2, 2), device="cuda")
    want = (ck.pack_weight_convT_fwd(wt), ck.pack_weight_convT_dgrad(wt))
    for both in ((True, True), (True, False), (False, True)):
        for got, ref, asked in zip(ck.pack_convT(wt, *both), want, both):
            assert torch.equal(got, ref) if asked else got is None
    w1 = torch.randn((cout, cin, 1, 1, 1), device="cuda")
    assert torch.equal(ck.pack_point(w1, ck.pad_channels(cin), False), ck.pack_weight_fwd(w1))
    assert torch.equal(ck.pack_point(w1, ck.pad_channels(cin), True), ck.pack_weight_dgrad(w1))
