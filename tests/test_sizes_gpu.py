"""Tensors that do not hold what a call reads of them are refused before anything is launched."""
import pytest
import torch

import haste_b200
from haste_b200 import _C, ops

pytestmark = pytest.mark.gpu
T, N, C, H = 5, 3, 12, 16
CELLS = ["LSTM", "GRU", "IndRNN", "LayerNormLSTM", "LayerNormGRU", "LayerNormIndRNN"]


def _refused(call):
    n0 = _C.launch_count()
    with pytest.raises(RuntimeError):
        call()
    assert _C.launch_count() == n0


@pytest.mark.parametrize("general", [False, True], ids=["compiled", "autograd functions"])
@pytest.mark.parametrize("cell", CELLS)
def test_layer_call(cell, general):
    layer = getattr(haste_b200, cell)(C, H, zoneout=0.1).cuda()
    if general:
        layer._native_applies = lambda *a: False
    x = torch.randn(T, N, C, device="cuda")
    mask = torch.ones(T, N, H, device="cuda")
    layer(x, zoneout_mask=mask)
    _refused(lambda: layer(x[:, :, :-1]))
    _refused(lambda: layer(x, zoneout_mask=mask[:-1]))
    _refused(lambda: layer(x, zoneout_mask=mask[:, :, :-1]))
    for name, p in list(layer.named_parameters()):
        if name == "gamma" and cell == "LayerNormIndRNN":
            continue  # the second row takes no part
        p.data, whole = p.data[..., :-1].contiguous(), p.data
        _refused(lambda: layer(x, zoneout_mask=mask))
        p.data = whole
    layer(x, zoneout_mask=mask)


def test_backward_op():
    new = lambda *s: torch.randn(*s, device="cuda")
    x, W, R, b, none = new(T, N, C), new(C, 4 * H), new(H, 4 * H), new(4 * H), new(0, 0, 0)
    h, c, cache = ops.lstm_forward(True, 0.0, x, new(N, H), new(N, H), W, R, b, none)
    args = [x, W, R, b, none, h, c, cache, new(T + 1, N, H), new(T + 1, N, H)]
    for i in (0, 1, 2, 4, 6, 7, 8, 9):
        short = list(args)
        short[i] = new(T, N, H - 1) if i == 4 else args[i][1:].contiguous()
        _refused(lambda: ops.lstm_backward(*short, transposed=False))
    ops.lstm_backward(*args, transposed=False)
