"""Operator behaviour that is decided on the host before any device is needed."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from flashbias_b200 import FlashBiasAlibiFunc, FlashBiasFunc, flash_bias_alibi_func, flash_bias_func


@pytest.mark.parametrize("with_grad", [False, True])
@pytest.mark.parametrize("which", range(6))
def test_tangents_are_refused_and_not_dropped(which, with_grad):
    t = [torch.randn(1, 16, 2, 8).half() for _ in range(3)] + [torch.randn(1, 16, 2, 4).half() for _ in range(2)]
    t.append(torch.zeros(1, 1, 16, 16))
    t[0].requires_grad_(with_grad)
    with fwAD.dual_level():
        t[which] = fwAD.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            flash_bias_func(*t)


@pytest.mark.parametrize("which", range(4))
def test_tangents_are_refused_by_the_slope_form(which):
    t = [torch.randn(1, 16, 2, 8).half() for _ in range(3)] + [torch.ones(2)]
    with fwAD.dual_level():
        t[which] = fwAD.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            flash_bias_alibi_func(*t)


@pytest.mark.parametrize("cls", [FlashBiasFunc, FlashBiasAlibiFunc])
def test_operators_are_autograd_functions(cls):
    assert issubclass(cls, torch.autograd.Function)
    for name in ("forward", "backward"):
        assert name in cls.__dict__
