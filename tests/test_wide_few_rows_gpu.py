"""Exactness of wide fp32 layers of few rows, against fp64."""
import pytest
import torch

import haste_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,N,H", [("LSTM", 16, 640), ("LSTM", 60, 520), ("GRU", 31, 768), ("GRU", 8, 1024)])
def test_wide_layers_of_few_rows_are_as_exact_as_step_by_step(cell, N, H):
    """fp32, beyond 512 units, where the step-wise path would use fp32 FMAs: the relative error of the
    output against fp64 is no larger than by that path (4.5e-6, what two planes leave in x.W)."""
    import haste_b200
    torch.manual_seed(H)
    T, C = 60, 96
    layer = getattr(haste_b200, cell)(C, H).cuda()
    with torch.no_grad():
        layer.recurrent_kernel.normal_(0.0, H ** -0.5)
    x = torch.randn(T, N, C, device="cuda")
    d = lambda t: t.detach().double()
    zero = x.new_zeros(N, H, dtype=torch.float64)
    if cell == "LSTM":
        want = oracle.lstm(True, 0.0, d(x), zero, zero, d(layer.kernel), d(layer.recurrent_kernel), d(layer.bias))[0]
    else:
        want = oracle.gru(True, 0.0, d(x), zero, d(layer.kernel), d(layer.recurrent_kernel), d(layer.bias),
                          d(layer.recurrent_bias))
    y = layer(x)[0]
    assert (d(y) - want[1:]).norm() < 4.5e-6 * want[1:].norm()
