"""LayerNorm recurrences on clusters: the edges of their tiles against the fp64 oracle."""
import pytest
import torch

import haste_oracle as oracle
from helpers import TOL_BF16, TOL_F32, assert_close, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N,H", [(1, 1, 3), (3, 8, 16), (5, 9, 17), (6, 3, 64), (5, 17, 100), (4, 70, 128),
                                   (7, 33, 200), (4, 130, 250), (6, 8, 256),
                                   (5, 9, 257), (4, 70, 301), (6, 3, 320)])
@pytest.mark.parametrize("cell", ["layer_norm_lstm", "layer_norm_gru"])
def test_tiles_f32(cell, T, N, H):
    d = oracle.make_inputs(cell, T, N, 12, H, seed=H + N, zoneout=0.2)
    ref_out, ref_g = oracle.forward_backward(cell, d, zoneout=0.2)
    out, g = run_cuda(cell, d, zoneout=0.2)
    assert_close(out["h"], ref_out["h"], TOL_F32, "h")
    for k, r in ref_g.items():
        assert_close(g[k], r, TOL_F32, "d" + k)


@pytest.mark.parametrize("N,H", [(9, 40), (20, 256), (11, 300)])
def test_tiles_bf16(N, H):
    d = oracle.make_inputs("layer_norm_gru", 5, N, 16, H, seed=H, zoneout=0.2)
    dq = {k: (v.to(torch.bfloat16).to(torch.float64) if v is not None else None) for k, v in d.items()}
    ref_out, ref_g = oracle.forward_backward("layer_norm_gru", dq, zoneout=0.2)
    out, g = run_cuda("layer_norm_gru", dq, zoneout=0.2, dtype=torch.bfloat16)
    assert_close(out["h"], ref_out["h"], TOL_BF16, "h")
    for k, r in ref_g.items():
        assert_close(g[k], r, TOL_BF16, "d" + k)
