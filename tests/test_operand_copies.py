"""Which parameter a layer's bf16 operand copies belong to (host side; the packing kernel is replaced by a recorder)."""
import copy

import pytest
import torch

from scaffold_b200.ops import conv3d as c3
from scaffold_b200.ops.conv3d import Conv3d


@pytest.fixture
def packed(monkeypatch):
    calls = []
    monkeypatch.setattr(c3.ck, "pack_conv3", lambda w, *a: calls.append(w))
    return calls


def _use(conv):
    return conv._cache.conv3(conv.weight, [16], [16], "fwd", False)


def test_copies_are_made_once_per_weight_version(packed):
    conv = Conv3d(16, 16, 3, padding=1)
    _use(conv), _use(conv)
    assert len(packed) == 1
    with torch.no_grad():
        conv.weight.add_(1.0)
    _use(conv)
    assert len(packed) == 2


@pytest.mark.parametrize("how", ["deepcopy", "assign", "new_parameter"])
def test_copies_follow_another_parameter(packed, how):
    conv = Conv3d(16, 16, 3, padding=1)
    _use(conv)
    old = conv.weight
    generation = c3._PACK_GENERATION[0]
    if how == "deepcopy":
        conv = copy.deepcopy(conv)
    elif how == "assign":
        conv.load_state_dict({k: v.clone() for k, v in conv.state_dict().items()}, assign=True)
    else:
        conv.weight = torch.nn.Parameter(old.detach())  # the same memory
    assert conv.weight is not old
    _use(conv)
    assert packed[-1] is conv.weight and len(packed) == 2
    assert conv._cache._w_ref() is conv.weight and conv._cache in c3._PACK_REGISTRY
    assert c3._PACK_GENERATION[0] > generation
