"""The fused loss kernels against fp64 at the edges of their class tiles and with ragged voxel counts (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes,shape,weighted", [
    (2, (1, 1, 1, 1), False), (4, (2, 3, 5, 7), True), (5, (1, 8, 16, 8), False), (9, (3, 9, 11, 13), True),
    (12, (2, 4, 4, 33), False), (13, (1, 5, 6, 7), True), (17, (2, 16, 16, 17), False), (32, (1, 40, 64, 65), True)])
def test_fused_loss_matches_fp64(classes, shape, weighted):
    from scaffold_b200.ops import _lib, loss as L
    g = torch.Generator(device="cuda").manual_seed(classes)
    pad = (classes + 15) // 16 * 16
    logits = (torch.randn((*shape, pad), generator=g, device="cuda") * 3).to(torch.bfloat16)
    labels = torch.randint(0, classes, shape, generator=g, device="cuda", dtype=torch.int16)
    cw = torch.rand(classes, generator=g, device="cuda") + 0.5 if weighted else None
    ours = logits.clone().requires_grad_()
    loss, ce, fg = L.segmentation_loss_fused(ours, labels, classes, cw)
    (loss * 1.7).backward()
    ref = logits[..., :classes].double().permute(0, 4, 1, 2, 3).contiguous().requires_grad_()
    lp = torch.log_softmax(ref, 1)
    rce = L.sharded_cross_entropy(lp, labels, None if cw is None else cw.double())
    rfg = L.sharded_dice(lp.exp(), L.labels_to_onehot(labels, classes).double())[:, 1:].mean()
    ((rce + 1 - rfg) * 1.7).backward()
    _lib.check_status()
    # every term carries the error of one exponential and one logarithm (a few 2^-23 of values up to about 30) and the
    # sums are fp32 trees of at most 15 levels per thread and 20 across: 1e-5 of the value
    for a, b in ((ce, rce), (fg, rfg), (loss, rce + 1 - rfg)):
        assert abs(float(a.detach()) - float(b.detach())) <= 1e-5 * max(1.0, abs(float(b.detach())))
    gr = ref.grad.permute(0, 2, 3, 4, 1)
    got = ours.grad[..., :classes].double()
    # bf16 output: half a unit in the last place (2^-9) of the value, plus fp32 error of terms that may cancel
    terms = (1.7 / labels.numel() * (cw.max() if weighted else 1.0)) * 4 + 4 * gr.abs().amax()
    assert ((got - gr).abs() <= 2 ** -8 * gr.abs() + 1e-5 * terms).all()
    assert not ours.grad[..., classes:].any()


@pytest.mark.parametrize("classes,shape", [(3, (2, 7, 9, 11)), (9, (1, 32, 32, 33)), (32, (2, 4, 8, 16))])
def test_hard_dice_matches_the_formula(classes, shape):
    from scaffold_b200.ops import loss as L
    g = torch.Generator(device="cuda").manual_seed(7)
    pad = (classes + 15) // 16 * 16
    logits = torch.randint(-4, 5, (*shape, pad), generator=g, device="cuda").to(torch.bfloat16)  # many ties: first wins
    labels = torch.randint(0, max(2, classes - 1), shape, generator=g, device="cuda", dtype=torch.int32)
    got = L.hard_dice_fused(logits, labels, classes)
    ref = L.hard_dice_reference(logits[..., :classes].permute(0, 4, 1, 2, 3).float(), labels, classes)
    torch.testing.assert_close(got, ref, rtol=2e-7, atol=0)  # counts are exact; one quotient in fp32


def test_the_loss_can_be_changed_in_place():
    """The three results are tensors of their own, as the formula's are (gradient accumulation: ``loss /= n``)."""
    from scaffold_b200.ops import loss as L
    g = torch.Generator(device="cuda").manual_seed(1)
    logits = torch.randn((2, 4, 5, 6, 16), generator=g, device="cuda").to(torch.bfloat16)
    labels = torch.randint(0, 5, (2, 4, 5, 6), generator=g, device="cuda", dtype=torch.int16)
    a, b = logits.clone().requires_grad_(), logits.clone().requires_grad_()
    loss, ce, fg = L.segmentation_loss_fused(a, labels, 5, None)
    values = float(ce.detach()), float(fg.detach())
    loss /= 4
    loss.mul_(3.0).add_(1.0)
    loss.backward()
    ref, *_ = L.segmentation_loss_fused(b, labels, 5, None)
    (ref / 4 * 3.0 + 1.0).backward()
    assert torch.equal(loss, ref / 4 * 3.0 + 1.0) and torch.equal(a.grad, b.grad)
    assert (float(ce.detach()), float(fg.detach())) == values and not (loss._is_view() or ce._is_view() or fg._is_view())


def test_a_nan_class_weight_shows_in_every_gradient():
    """The cross-entropy's denominator is NaN then, for the voxels of the other classes too."""
    from scaffold_b200.ops import loss as L
    g = torch.Generator(device="cuda").manual_seed(1)
    logits = torch.randn((2, 4, 5, 6, 16), generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    labels = torch.randint(0, 5, (2, 4, 5, 6), generator=g, device="cuda", dtype=torch.int16)
    weights = torch.ones(5, device="cuda")
    weights[2] = float("nan")
    loss, ce, fg = L.segmentation_loss_fused(logits, labels, 5, weights)
    loss.backward()
    assert loss.isnan() and ce.isnan() and fg.isfinite()
    assert logits.grad[..., :5].isnan().all()
