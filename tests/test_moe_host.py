"""Checks of FusedMoe that need no GPU: tensors that claim to be on one, and a block that only records that it was called."""
from types import SimpleNamespace

import pytest
import torch

from candle_vllm_b200 import moe
from candle_vllm_b200._lib import BackendError

H, I, E = 256, 256, 4


def _claims(dtype, shape, device):
    numel = 1
    for n in shape:
        numel *= n
    return SimpleNamespace(dtype=dtype, shape=shape, device=torch.device(device), is_cuda=device != "cpu", dim=lambda: len(shape), numel=lambda: numel,
                           is_contiguous=lambda: True, contiguous=lambda: None, data_ptr=lambda: 256)


def _op(monkeypatch, **devices):
    op = object.__new__(moe.FusedMoe)
    stack = lambda name: _claims(torch.uint8, (E * I * H // 256 * 144,), devices.get(name, "cuda:0"))
    op.gate = _claims(torch.float32, (E, H), devices.get("gate", "cuda:0"))
    op.ge, op.ue, op.de, op.types = stack("ge"), stack("ue"), stack("de"), (12, 12, 12)
    op.E, op.H, op.I, op.k, op.norm_topk_prob, op.routed_scaling_factor = E, H, I, 2, True, None
    monkeypatch.setattr(moe, "require_device", lambda: None)
    monkeypatch.setattr(moe.FusedMoe, "_block", lambda self, xs, T: "launched")
    return op


def test_all_on_one_device_takes_the_block(monkeypatch):
    assert _op(monkeypatch).forward(_claims(torch.float32, (3, H), "cuda:0")) == "launched"


@pytest.mark.parametrize("name", ["gate", "ge", "ue", "de"])
@pytest.mark.parametrize("device", ["cpu", "cuda:1"])
def test_a_tensor_elsewhere_is_refused(monkeypatch, name, device):
    with pytest.raises(BackendError, match=f"on {device}, the input on cuda:0"):
        _op(monkeypatch, **{name: device}).forward(_claims(torch.float32, (3, H), "cuda:0"))
