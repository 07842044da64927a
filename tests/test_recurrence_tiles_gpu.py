"""The persistent LSTM / GRU recurrences at the edges of their tiles, against the CPU oracle:
hidden sizes on both sides of every change of tiling, batches that leave a chain of eight rows
partly empty or give a CTA several chains, every storage type."""
import pytest
import torch

import haste_oracle as oracle
from helpers import TOL_BF16, TOL_F16, TOL_F32, assert_close, run_cuda

pytestmark = pytest.mark.gpu

# (T, N, H): cluster kernels (H <= 320)
CLUSTER = [(1, 1, 1), (5, 2, 15), (6, 8, 16), (6, 9, 17), (7, 3, 64), (5, 33, 72), (5, 17, 129),
           (6, 7, 200), (6, 37, 250), (5, 64, 256), (5, 5, 258), (5, 20, 320), (4, 150, 256),
           (4, 300, 320), (3, 700, 64)]


def _check(cell, T, N, H, dtype, tol, zoneout, transposed=False):
    d = oracle.make_inputs(cell, T, N, 12, H, seed=T * 1000 + H + N, zoneout=zoneout)
    dq = {k: (v.to(dtype).to(torch.float64) if v is not None else None) for k, v in d.items()}
    ref_out, ref_grads = oracle.forward_backward(cell, dq, zoneout=zoneout)
    out, grads = run_cuda(cell, dq, zoneout=zoneout, dtype=dtype, transposed=transposed)
    for k, ref in list(ref_out.items()) + list(ref_grads.items()):
        if k in out or k in grads:
            assert_close(out[k] if k in out else grads[k], ref, tol, f"{cell} {k}")


@pytest.mark.parametrize("zoneout", [0.0, 0.25])
@pytest.mark.parametrize("shape", CLUSTER, ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_cluster_recurrence_fp32(cell, shape, zoneout):
    _check(cell, *shape, torch.float32, TOL_F32, zoneout, transposed=shape[1] % 2 == 0)


@pytest.mark.parametrize("shape", [(5, 9, 17), (6, 37, 250), (5, 20, 320), (4, 150, 256)],
                         ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell,dtype,tol", [("lstm", torch.bfloat16, TOL_BF16),
                                            ("gru", torch.bfloat16, TOL_BF16),
                                            ("gru", torch.float16, TOL_F16)])
def test_cluster_recurrence_reduced_precision(cell, dtype, tol, shape):
    _check(cell, *shape, dtype, tol, 0.25)


# (T, N, H): grid kernels - every tiling of the hidden dimension, several chains per CTA
GRID = [(5, 9, 321), (4, 20, 388), (5, 70, 512), (8, 1, 516), (8, 33, 520), (8, 12, 760),
        (8, 17, 1020), (8, 9, 1024), (4, 300, 200)]


@pytest.mark.parametrize("zoneout", [0.0, 0.25])
@pytest.mark.parametrize("shape", GRID, ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_grid_recurrence_fp32(cell, shape, zoneout):
    _check(cell, *shape, torch.float32, TOL_F32, zoneout, transposed=shape[1] % 2 == 0)


@pytest.mark.parametrize("shape", [(5, 9, 321), (8, 33, 520), (8, 17, 1020), (8, 70, 1024)],
                         ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell,dtype,tol", [("lstm", torch.bfloat16, TOL_BF16),
                                            ("gru", torch.bfloat16, TOL_BF16),
                                            ("gru", torch.float16, TOL_F16)])
def test_grid_recurrence_reduced_precision(cell, dtype, tol, shape):
    _check(cell, *shape, dtype, tol, 0.25)


@pytest.mark.parametrize("shape", [(1, 3, 513), (2, 64, 640), (4, 6, 1024), (7, 17, 900)],
                         ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_short_sequences_of_wide_layers_take_the_recurrence(cell, shape):
    """A few steps of an fp32 layer beyond 512 units: right, and one launch for the recurrence of
    each pass, so that the launches do not grow with the steps."""
    from haste_b200 import _C
    n0 = _C.launch_count()
    _check(cell, *shape, torch.float32, TOL_F32, 0.25)
    assert _C.launch_count() - n0 <= 14


# tensor-core recurrence: two 64-row tiles per CTA with a ragged second one, a last slice of eight units, rings whose stage
# count is no multiple of the issuers, fewer k-blocks than issuers have turns
@pytest.mark.parametrize("T,N,H,sms", [(40, 90, 1024, 74), (40, 65, 1024, 74), (60, 128, 768, 74), (8, 700, 320, 0),
                                        (20, 90, 1000, 74), (8, 700, 328, 0), (12, 130, 808, 74)])
@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_tensor_core_tiles(cell, T, N, H, sms):
    from haste_b200 import _C
    _C.set_sm_budget(sms)
    try:
        _check(cell, T, N, H, torch.bfloat16, TOL_BF16, 0.25, transposed=N % 4 == 0)
        _C.sync_check(torch.cuda.current_stream().cuda_stream)
    finally:
        _C.set_sm_budget(0)


@pytest.mark.parametrize("N,H", [(64, 1024), (90, 1000), (128, 768)])
def test_tensor_core_gru_gates_are_exact(N, H):
    """One step from each stored state in fp64, rounded to bf16: gate functions good to 1e-6 leave
    another bf16 in 0.02 % of the values, one MUFU.TANH each (2^-11) in 0.17 %."""
    import haste_b200
    torch.manual_seed(1)
    T, C = 30, 128
    layer = haste_b200.GRU(C, H).cuda().bfloat16()
    layer._sm_budget = 74  # of the GPU: every case takes the tensor-core recurrence
    with torch.no_grad():
        layer.recurrent_kernel.normal_(0.0, H ** -0.5)
        x = torch.randn(T, N, C, device="cuda").bfloat16()
        y = layer(x)[0]
        W, R, b, br = [p.double() for p in layer.parameters()]
        h = torch.cat([torch.zeros_like(y[:1]), y[:-1]]).double()
        zx, rx, gx = ((x.double() @ W).bfloat16().double() + b).chunk(3, 2)
        zh, rh, gh = (h @ R + br).chunk(3, 2)
        z, r = (zx + zh).sigmoid(), (rx + rh).sigmoid()
        want = (z * h + (1 - z) * (gx + r * gh).tanh()).bfloat16()
    assert (y != want).double().mean() < 6e-4


# beyond 512 units with more rows: sixteen units per CTA, R's second plane in shared memory
@pytest.mark.parametrize("shape", [(5, 24, 513), (6, 31, 1024), (5, 45, 777), (4, 64, 640), (4, 100, 530), (3, 190, 1021)],
                         ids=lambda s: "T%d_N%d_H%d" % s)
@pytest.mark.parametrize("cell,dtype,tol", [("lstm", torch.float32, TOL_F32), ("gru", torch.float32, TOL_F32),
                                            ("gru", torch.float16, TOL_F16)])
@pytest.mark.parametrize("budget", [0, 74])
def test_grid_recurrence_of_wide_layers(cell, dtype, tol, shape, budget):
    from haste_b200 import _C
    was = _C.exchange_sm_budget(budget)
    try:
        _check(cell, *shape, dtype, tol, 0.25, transposed=shape[1] % 2 == 0)
    finally:
        _C.exchange_sm_budget(was)


def test_few_rows_do_not_go_to_the_tensor_cores():
    """Two chains of eight rows per CTA are far ahead of a tile of 64 (1.9 and 6.8 us per step)."""
    import haste_b200
    from torch.profiler import ProfilerActivity, profile
    for cell in (haste_b200.LSTM, haste_b200.GRU):
        layer = cell(64, 512).cuda().bfloat16()
        x = torch.randn(3, 64, 64, device="cuda").bfloat16()
        with profile(activities=[ProfilerActivity.CUDA]) as seen:
            layer(x)[0].float().sum().backward()
            torch.cuda.synchronize()
        assert not [e.name for e in seen.events() if "tc_recurrence" in e.name]


# a quarter of K per CTA of a cluster: two 128-row and two 64-row tiles per CTA, one of either, unequal shares of K, a
# cluster with units beyond H
@pytest.mark.parametrize("T,N,H,sms", [(6, 256, 1024, 74), (5, 200, 520, 74), (5, 190, 688, 74), (4, 300, 1016, 0),
                                        (3, 270, 744, 74), (4, 128, 1024, 0)])
@pytest.mark.parametrize("cell", ["lstm", "gru"])
def test_tensor_core_backward_shares_out_k(cell, T, N, H, sms):
    from haste_b200 import _C
    _C.set_sm_budget(sms)
    try:
        _check(cell, T, N, H, torch.bfloat16, TOL_BF16, 0.25, transposed=N % 4 == 0)
        _C.sync_check(torch.cuda.current_stream().cuda_stream)
    finally:
        _C.set_sm_budget(0)
