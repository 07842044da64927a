"""Contractions whose rows are not multiples of 16 bytes: operands go through a copy, results
leave value by value."""
import pytest
import torch

from haste_b200 import _C, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("M,K,N", [(64, 67, 513), (333, 161, 750), (200, 1999, 33), (1000, 64, 161), (65, 515, 193)])
@pytest.mark.parametrize("transposed", [False, True])
def test_odd_leading_dimensions(M, K, N, transposed, dtype, tol):
    torch.manual_seed(M + N)
    a = torch.randn(K, M, device="cuda").to(dtype).t() if transposed else torch.randn(M, K, device="cuda").to(dtype)
    b = torch.randn(K, N, device="cuda").to(dtype)
    c = torch.randn(M, N, device="cuda").to(dtype)
    want = a.double() @ b.double()
    _C.set_gemm_path(_C.GEMM_TCGEN05)
    try:
        got = ops.gemm(a, b)
        added = ops.gemm(a, b, out=c.clone(), accumulate=True)
    finally:
        _C.set_gemm_path(_C.GEMM_AUTO)
    scale = want.abs().max().item()
    assert (got.double() - want).abs().max().item() < tol * scale
    assert (added.double() - want - c.double()).abs().max().item() < tol * scale


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,H", [(1, 1, 1), (8, 2, 5), (17, 3, 64), (9, 40, 1024), (20, 100, 1000)])
def test_column_sums_and_scans(T, N, H, dtype):
    """IndRNN gradients at the edges of the scan's groups of steps and of the column sums."""
    import haste_oracle as oracle
    from helpers import TOL_BF16, TOL_F32, assert_close, run_cuda
    d = oracle.make_inputs("indrnn", T, N, 8, H, seed=T + H, zoneout=0.2)
    if dtype == torch.bfloat16:
        d = {k: (v.to(dtype).to(torch.float64) if v is not None else None) for k, v in d.items()}
    ref_out, ref_g = oracle.forward_backward("indrnn", d, zoneout=0.2)
    out, g = run_cuda("indrnn", d, zoneout=0.2, dtype=dtype)
    tol = TOL_F32 if dtype == torch.float32 else TOL_BF16
    assert_close(out["h"], ref_out["h"], tol, "h")
    for k, r in ref_g.items():
        assert_close(g[k], r, tol, "d" + k)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("M,K,N", [(8, 512, 2048), (16, 512, 2048), (24, 6400, 1024), (31, 1999, 193), (31, 67, 2051)])
@pytest.mark.parametrize("transposed", [False, True])
def test_few_rows_are_fp32_grade(M, K, N, transposed, dtype):
    """Fewer than 32 rows: as exact as fp32 FMAs.  Bound: products dropped below 2^-24, fp32 sums of
    chunks, an fp32 (fp16) result: 1e-6 (2^-11) of the result in the 2-norm; two planes leave 4e-6."""
    torch.manual_seed(M + N)
    a = torch.randn(K, M, device="cuda").to(dtype).t() if transposed else torch.randn(M, K, device="cuda").to(dtype)
    b = torch.randn(K, N, device="cuda").to(dtype)
    want = a.double() @ b.double()
    got = ops.gemm(a, b).double()
    bound = 1e-6 if dtype == torch.float32 else 2.0 ** -11
    assert (got - want).norm() < bound * want.norm()


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("M,K,N", [(2048, 20000, 3072), (2000, 8200, 2601), (5000, 8192, 900)])
def test_long_sums_over_more_than_one_wave(M, K, N, dtype, tol):
    """Weight gradients of wide layers: more tiles than the GPU holds at once, K split all the same.  The bounds
    are those of the edges above."""
    torch.manual_seed(K)
    a, b = torch.randn(K, M, device="cuda").to(dtype).t(), torch.randn(K, N, device="cuda").to(dtype)
    c = torch.randn(M, N, device="cuda").to(dtype)
    want = a.double() @ b.double()
    scale = want.abs().max().item()
    assert (ops.gemm(a, b).double() - want).abs().max().item() < tol * scale
    added = ops.gemm(a, b, out=c.clone(), accumulate=True)
    assert (added.double() - want - c.double()).abs().max().item() < tol * scale


@pytest.mark.parametrize("M", [32, 33, 63, 64, 65])
@pytest.mark.parametrize("K,N", [(512, 2048), (1100, 130), (2048, 1027)])
def test_partial_tiles_of_few_rows(M, K, N):
    """Up to 64 rows partial tiles leave from the lanes, beyond through shared memory; the bound is that of the edges above."""
    torch.manual_seed(M + N)
    a, b = torch.randn(M, K, device="cuda"), torch.randn(K, N, device="cuda")
    want = a.double() @ b.double()
    c = torch.randn(M, N, device="cuda")
    scale = want.abs().max().item()
    assert (ops.gemm(a, b).double() - want).abs().max().item() < 2e-5 * scale
    added = ops.gemm(a, b, out=c.clone(), accumulate=True)
    assert (added.double() - want - c.double()).abs().max().item() < 2e-5 * scale
