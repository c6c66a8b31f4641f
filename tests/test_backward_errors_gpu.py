"""Exceptions of a backward pass, which runs on a thread of the autograd engine."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _x(K, T=64):
    return torch.randn(1, T, 2, K, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").to(torch.bfloat16) / K ** 0.5


def test_the_device_error_word_is_read_when_asked_for(monkeypatch):
    from tops_b200 import _lib as L
    from tops_b200.ops.gla import chunk_gla
    x = _x(128)
    leaf = x.clone().requires_grad_()
    monkeypatch.setattr(L, "CHECK_DEVICE", True)
    o = chunk_gla(leaf, x, x, -x.abs())[0]
    L.check(L.lib.tops_b200_device_error_set(7), "device_error_set")
    with pytest.raises(L.TopsError, match="code 7"):
        o.backward(x)
    assert L.device_error() == 0   # the word is cleared by the error it raises
    o = chunk_gla(leaf, x, x, -x.abs())[0]
    o.backward(x)
    monkeypatch.setattr(L, "CHECK_DEVICE", False)
    L.check(L.lib.tops_b200_device_error_set(7), "device_error_set")
    try:
        chunk_gla(leaf, x, x, -x.abs())[0].backward(x)
    finally:
        L.device_error_reset()


def test_what_a_backward_refuses_is_an_assertion():
    from tops_b200.ops.kda import fused_recurrent_kda
    x = _x(192, 3).requires_grad_()
    o = fused_recurrent_kda(x, x, x, -x.abs(), x[..., 0].sigmoid())[0]
    with pytest.raises(AssertionError, match="K, V <= 128"):
        o.sum().backward()
