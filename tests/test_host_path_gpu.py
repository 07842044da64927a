"""The layers' compiled host path against the autograd functions over the tensor-level ops."""
import pytest
import torch

import haste_b200

pytestmark = pytest.mark.gpu
CELLS = ["LSTM", "GRU", "IndRNN", "LayerNormLSTM", "LayerNormGRU", "LayerNormIndRNN"]


def _leaves(state):
    return list(state) if isinstance(state, tuple) else [state]


def _run(layer, x, state, loss, general, **kw):
    if general:
        layer._native_applies = lambda *a: False
    leaves = [x] + (_leaves(state) if state is not None else []) + list(layer.parameters())
    leaves = [t for t in leaves if t.requires_grad]
    y, final = layer(x, state, **kw)
    out = [y] + _leaves(final)
    grads = torch.autograd.grad(loss(y, _leaves(final)), leaves, allow_unused=True) if loss else []
    layer.__dict__.pop("_native_applies", None)
    return out + list(grads)


LOSSES = {"output": lambda y, s: (y * y).sum(), "state": lambda y, s: sum((t * t).sum() for t in s),
          "both": lambda y, s: y.sum() + (s[-1] * s[-1]).sum()}


@pytest.mark.parametrize("loss", sorted(LOSSES))
@pytest.mark.parametrize("T,N,C,H,batch_first,sequence,given,dx", [
    (1, 1, 1, 1, False, False, False, True), (1, 4, 24, 32, False, False, True, False),
    (9, 5, 19, 33, True, False, True, True), (6, 8, 32, 64, False, True, False, False)])
@pytest.mark.parametrize("cell", CELLS)
def test_training_call(cell, T, N, C, H, batch_first, sequence, given, dx, loss):
    torch.manual_seed(T + H)
    layer = getattr(haste_b200, cell)(C, H, batch_first=batch_first, zoneout=0.2,
                                      return_state_sequence=sequence).cuda()
    x = torch.randn(N if batch_first else T, T if batch_first else N, C, device="cuda", requires_grad=dx)
    state = None
    if given:
        state = torch.randn(1, N, H, device="cuda", requires_grad=True)
        if "LSTM" in cell:
            state = (state, torch.randn(1, N, H, device="cuda", requires_grad=True))
    mask = torch.empty(T, N, H, device="cuda").bernoulli_(0.8)
    got, want = [_run(layer, x, state, LOSSES[loss], g, zoneout_mask=mask) for g in (False, True)]
    for a, b in zip(got, want):
        assert a.shape == b.shape
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,H,zoneout", [(1, 1, 8, 0.0), (1, 33, 72, 0.1), (7, 3, 40, 0.1)])
@pytest.mark.parametrize("cell", CELLS)
def test_inference_call(cell, T, N, H, zoneout, dtype):
    torch.manual_seed(N)
    layer = getattr(haste_b200, cell)(16, H, zoneout=zoneout).cuda().to(dtype).eval()
    x = torch.randn(T, N, 16, device="cuda", dtype=dtype)
    lengths = [t % (T + 1) for t in range(N)]  # 0: the state that the row began with
    state = torch.randn(1, N, H, device="cuda", dtype=dtype)
    state = (state, state * 2) if "LSTM" in cell else state
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    with torch.no_grad():
        for kw in ({}, {"lengths": lengths}):
            got, want = [_run(layer, x, state, None, g, **kw) for g in (False, True)]
            for a, b in zip(got, want):
                torch.testing.assert_close(a, b, rtol=tol, atol=tol)


def test_settings_of_the_caller_survive_a_call():
    from haste_b200 import _C
    exchange = _C.lib().haste_b200_exchange_assign_gradients
    layer = haste_b200.GRU(8, 16).cuda()
    layer._sm_budget = 74
    x = torch.randn(3, 2, 8, device="cuda", requires_grad=True)
    _C.set_sm_budget(100)
    exchange(1)
    try:
        layer(x)[0].sum().backward()  # (the backward pass runs on a thread of autograd's)
        assert _C.sm_budget() == 100
    finally:
        _C.set_sm_budget(0)
        assert exchange(0) == 1
