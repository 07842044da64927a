"""Tracing and forward-mode AD of a layer: refused, or right - never a result that silently lacks
the layer."""
import pytest
import torch
import torch.autograd.forward_ad as forward_ad

import haste_b200

pytestmark = pytest.mark.gpu
CELLS = ["LSTM", "GRU", "IndRNN", "LayerNormLSTM", "LayerNormGRU", "LayerNormIndRNN"]


@pytest.mark.parametrize("T", [1, 5])
@pytest.mark.parametrize("frozen", [False, True])
@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("cell", CELLS)
def test_forward_mode_is_refused(cell, training, frozen, T):
    layer = getattr(haste_b200, cell)(8, 16).cuda().train(training).requires_grad_(not frozen)
    x = torch.randn(T, 3, 8, device="cuda")
    with forward_ad.dual_level():
        layer(x)
        with pytest.raises(NotImplementedError):
            layer(forward_ad.make_dual(x, torch.ones_like(x)))
        with torch.no_grad(), pytest.raises(NotImplementedError):
            layer(forward_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("T", [1, 5])
@pytest.mark.parametrize("frozen", [False, True])
@pytest.mark.parametrize("cell", CELLS)
def test_trace(cell, frozen, T):
    layer = getattr(haste_b200, cell)(8, 16).cuda().eval().requires_grad_(not frozen)
    x, other = torch.randn(2, T, 3, 8, device="cuda")
    with torch.no_grad():
        try:
            traced = torch.jit.trace(lambda a: layer(a)[0], x, check_trace=False)
        except RuntimeError:
            return
        torch.testing.assert_close(traced(other), layer(other)[0])
