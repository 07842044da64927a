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


@pytest.mark.parametrize("cell", ["lstm", "gru", "indrnn", "layer_norm_lstm", "layer_norm_gru", "layer_norm_indrnn"])
def test_compiled_extension(cell):
    """haste_pytorch_lib: one tensor after another a value short (initial states are copied by torch,
    which checks them)."""
    import importlib.util
    import haste_oracle as oracle
    from haste_b200 import build
    spec = importlib.util.spec_from_file_location("haste_pytorch_lib", build.TORCH_EXT)
    lib = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(lib)
    d = oracle.make_inputs(cell, T, N, C, H, seed=1, zoneout=0.2)
    t = {k: v.float().cuda().contiguous() for k, v in d.items() if v is not None}
    has_c = "lstm" in cell
    names = {"lstm": ["W", "R", "b"], "gru": ["W", "R", "bx", "br"], "indrnn": ["W", "u", "b"],
             "layer_norm_lstm": ["W", "R", "b", "gamma", "gamma_h", "beta_h"],
             "layer_norm_gru": ["W", "R", "bx", "br", "gamma"], "layer_norm_indrnn": ["W", "u", "b", "gamma"]}[cell]
    forward, backward = getattr(lib, cell + "_forward"), getattr(lib, cell + "_backward")
    states = [t["h0"], t["c0"]] if has_c else [t["h0"]]
    fwd = [t["x"], *states, *[t[n] for n in names], t["mask"]]
    out = forward(True, 0.2, *fwd)
    out = list(out) if isinstance(out, (list, tuple)) else [out]
    turned = [t[n].t().contiguous() if n in ("W", "R") else t[n] for n in names]
    bwd = [t["x"].permute(2, 0, 1).contiguous(), *turned, t["mask"], *out, t["dh"]] + ([t["dc"]] if has_c else [])
    short = lambda a: a.reshape(-1)[:-1].clone().view(*([1] * (a.dim() - 1)), -1)
    read = lambda n: not (n == "gamma" and cell == "layer_norm_indrnn")
    for i, n in enumerate(names):
        if read(n) and n not in ("R", "u") and not (n == "W" and "indrnn" in cell):
            bad = list(fwd)
            bad[1 + len(states) + i] = short(bad[1 + len(states) + i])
            _refused(lambda: forward(True, 0.2, *bad))
    _refused(lambda: forward(True, 0.2, *fwd[:-1], short(fwd[-1])))
    for i in range(1, len(bwd)):
        n = names[i - 1] if i <= len(names) else ""
        h = len(names) + 2
        if i == h or not read(n) or n in ("b", "bx", "br"):
            continue  # the sizes come from h; biases are not read; the second row of gamma neither
        bad = list(bwd)
        bad[i] = short(bad[i])
        _refused(lambda: backward(*bad))
    backward(*bwd)
