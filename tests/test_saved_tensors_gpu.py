"""What a layer keeps for its backward pass, where something stands between saving and use."""
import pytest
import torch
from torch.autograd.graph import save_on_cpu, saved_tensors_hooks
from torch.utils.checkpoint import checkpoint

import haste_b200

pytestmark = pytest.mark.gpu
CELLS = ["LSTM", "GRU", "IndRNN", "LayerNormLSTM", "LayerNormGRU", "LayerNormIndRNN"]


def _case(cell, dtype=torch.float32):
    torch.manual_seed(3)
    T, N, C, H = 6, 5, 12, 24
    layer = getattr(haste_b200, cell)(C, H, zoneout=0.2).cuda().to(dtype)
    x = torch.randn(T, N, C, device="cuda", dtype=dtype, requires_grad=True)
    state = torch.randn(1, N, H, device="cuda", dtype=dtype, requires_grad=True)
    leaves = [x, state] + list(layer.parameters())
    if "LSTM" in cell:
        second = torch.randn(1, N, H, device="cuda", dtype=dtype, requires_grad=True)
        leaves.append(second)
        state = (state, second)
    mask = torch.empty(T, N, H, device="cuda", dtype=dtype).bernoulli_(0.8)
    return layer, x, state, mask, leaves


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cell", CELLS)
def test_hooks_and_checkpointing(cell, dtype):
    layer, x, state, mask, leaves = _case(cell, dtype)
    call = lambda a: layer(a, state, zoneout_mask=mask)[0]
    loss = lambda y: (y.float() * y.float()).sum()
    want = torch.autograd.grad(loss(call(x)), leaves)
    # an unpacked copy stands alone in its buffer, with other values around it
    fresh = lambda t: torch.full((3,) + tuple(t.shape), 7.0, device=t.device, dtype=t.dtype)

    def unpack(t):
        room = fresh(t)
        room[1] = t
        return room[1]

    for context in (lambda: save_on_cpu(), lambda: saved_tensors_hooks(lambda t: t.clone(), unpack)):
        with context():
            y = call(x)
        got = torch.autograd.grad(loss(y), leaves)
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    got = torch.autograd.grad(loss(checkpoint(call, x, use_reentrant=False)), leaves)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cell", CELLS)
def test_a_change_of_the_output_in_place_is_noticed(cell):
    layer, x, state, mask, leaves = _case(cell)
    y, _ = layer(x, state, zoneout_mask=mask)
    y.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y.sum(), leaves)


def test_a_hook_that_returns_another_type_is_refused():
    layer, x, state, mask, leaves = _case("LSTM")
    with saved_tensors_hooks(lambda t: t.half(), lambda t: t):
        y, _ = layer(x, state, zoneout_mask=mask)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y.sum(), leaves)
