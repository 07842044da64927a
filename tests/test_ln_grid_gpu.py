"""LayerNorm recurrences over the whole grid (beyond 320 units, or many rows): the edges of their tiles,
chains and scales against the fp64 oracle."""
import pytest
import torch

import haste_oracle as oracle
from haste_b200 import _C
from helpers import TOL_BF16, TOL_BF16_ALL_STORAGE_LN_LSTM, TOL_F32, assert_close, run_cuda

pytestmark = pytest.mark.gpu


def check(cell, d, tol, dtype=torch.float32, grad=1.0):
    if dtype == torch.bfloat16:
        d = {k: (v.to(dtype).to(torch.float64) if v is not None else None) for k, v in d.items()}
    ref_out, ref_g = oracle.forward_backward(cell, d, zoneout=0.2)
    out, g = run_cuda(cell, d, zoneout=0.2, dtype=dtype)
    assert_close(out["h"], ref_out["h"], tol, "h")
    for k, r in ref_g.items():
        assert_close(g[k].double() / grad, r / grad, tol, "d" + k)


# slices of 16 units with a ragged last one, rows that are no multiple of 4, one to eight chains per CTA
@pytest.mark.parametrize("T,N,H", [(1, 1, 321), (2, 8, 336), (5, 9, 353), (6, 3, 384), (4, 17, 400), (5, 33, 497),
                                   (7, 41, 510), (4, 70, 512), (3, 130, 511), (3, 250, 512), (4, 150, 300)])
@pytest.mark.parametrize("cell", ["layer_norm_lstm", "layer_norm_gru"])
def test_tiles_f32(cell, T, N, H):
    check(cell, oracle.make_inputs(cell, T, N, 12, H, seed=H + N, zoneout=0.2), TOL_F32)


# half of the GPU, and one row group of many chains (fewer slots for partial tiles than chains)
@pytest.mark.parametrize("budget,N,H", [(74, 64, 512), (74, 100, 340), (40, 60, 512), (33, 64, 500), (24, 50, 370)])
@pytest.mark.parametrize("cell", ["layer_norm_lstm", "layer_norm_gru"])
def test_sm_budget(cell, budget, N, H):
    was = _C.exchange_sm_budget(budget)
    try:
        check(cell, oracle.make_inputs(cell, 5, N, 12, H, seed=H, zoneout=0.2), TOL_F32)
    finally:
        _C.exchange_sm_budget(was)


# states of 2 and more take a scale of their own; gradients of any size take theirs from a bound
@pytest.mark.parametrize("state,grad", [(1.0, 1e-12), (3.0, 1.0), (500.0, 1e9), (1e-4, 1.0)])
@pytest.mark.parametrize("cell", ["layer_norm_lstm", "layer_norm_gru"])
def test_scales(cell, state, grad):
    d = oracle.make_inputs(cell, 4, 21, 12, 400, seed=7, zoneout=0.2)
    d["h0"] = d["h0"] * state
    d["h0"][3] = 0.0
    for k in ("dh", "dc"):
        if k in d:
            d[k] = d[k] * grad
    check(cell, d, TOL_F32, grad=grad)


@pytest.mark.parametrize("N,H", [(9, 330), (20, 512), (13, 777), (70, 1000), (30, 1024)])
def test_tiles_bf16(N, H):
    check("layer_norm_gru", oracle.make_inputs("layer_norm_gru", 5, N, 16, H, seed=H, zoneout=0.2), TOL_BF16, torch.bfloat16)


# One row of a large state among ordinary ones: the others come out bit for bit as without it, and within the bar.
# (The forward pass alone: the large row's gradients are not finite beyond 1e19, and parameter gradients sum over rows.)
@pytest.mark.parametrize("large", [1e6, 1e9, 1e30, float("inf"), float("nan")])
@pytest.mark.parametrize("whole_row", [True, False])
@pytest.mark.parametrize("cell,N,H", [("layer_norm_lstm", 9, 400), ("layer_norm_gru", 21, 512), ("layer_norm_gru", 150, 300)])
def test_a_large_row_stays_to_itself(cell, N, H, whole_row, large):
    d = oracle.make_inputs(cell, 6, N, 12, H, seed=9, zoneout=0.2)
    d["h0"] = d["h0"].clamp(-1.5, 1.5)
    plain = run_cuda(cell, d, zoneout=0.2, backward=False)[0]["h"]
    d["h0"][5, slice(None) if whole_row else 37] = large
    got = run_cuda(cell, d, zoneout=0.2, backward=False)[0]["h"]
    others = [n for n in range(N) if n != 5]
    assert torch.equal(got[:, others], plain[:, others])
    ref = oracle.forward_backward(cell, d, zoneout=0.2)[0]["h"]
    assert_close(got[:, others], ref[:, others], TOL_F32, "h")


def test_the_first_step_takes_the_whole_initial_state():
    """Initial states 1 and 1 + 2^-23, R of one 1 per column: h.R is h0 itself, and a gain of 1000 over the root of
    LayerNorm's epsilon makes 0.038 of the last bit.  The row's mean may be off by 2^-22 (its words have 23 bits): 0.075 in all
    gates alike, which moves the slopes of sigmoid and tanh by less than a tenth."""
    cell, N, H = "layer_norm_gru", 3, 336
    d = oracle.make_inputs(cell, 1, N, 12, H, seed=1)
    for k in ("W", "bx", "br"):
        d[k] = torch.zeros_like(d[k])
    d["h0"] = (1 + 2.0 ** -23 * (torch.arange(H) % 2)).double().expand(N, H).contiguous()
    d["R"] = torch.eye(H, dtype=torch.float64).repeat(1, 3)
    d["gamma"] = torch.full_like(d["gamma"], 1000.0)
    step = lambda h: (h[1, :, 1::2].double().mean() - h[1, :, 0::2].double().mean()).item()
    want = step(oracle.forward_backward(cell, d)[0]["h"])
    got = step(run_cuda(cell, d, backward=False)[0]["h"].cpu())
    assert abs(got - want) < 0.1 * abs(want)


# all-bf16 LayerNormLSTM: fragments of R in shared memory beyond 512 units, two statistic sources per lane, rows that
# start anywhere.  Against the oracle at that mode's bar, and against the step-wise path, which rounds tensors of
# the same kind and so lies within the same distance; a slip of layout is of order 1.
@pytest.mark.parametrize("N,H", [(9, 330), (13, 777), (70, 1000), (30, 1024)])
def test_tiles_bf16_lstm(N, H):
    d = oracle.make_inputs("layer_norm_lstm", 3, N, 16, H, seed=H, zoneout=0.2)
    d = {k: (v.to(torch.bfloat16).double() if v is not None else None) for k, v in d.items()}
    ref_out, ref_g = oracle.forward_backward("layer_norm_lstm", d, zoneout=0.2)
    run = lambda: run_cuda("layer_norm_lstm", d, zoneout=0.2, dtype=torch.bfloat16,
                           fwd_kwargs={"saved_dtype": torch.bfloat16})
    out, g = run()
    _C.set_recurrence_path(_C.PATH_STEPWISE)
    try:
        step_out, step_g = run()
    finally:
        _C.set_recurrence_path(_C.PATH_AUTO)
    bar = TOL_BF16_ALL_STORAGE_LN_LSTM
    assert_close(out["h"], ref_out["h"], bar, "h")
    assert_close(out["h"], step_out["h"], bar, "h, step by step")
    for k, r in ref_g.items():
        assert_close(g[k].double(), r, bar, "d" + k)
        assert_close(g[k].double(), step_g[k].double(), bar, "d%s, step by step" % k)
