"""Input projections of IndRNN and the LayerNorm cells that go through two scaled fp16 planes per operand
(large contractions): the saved x.W against float64."""
import pytest
import torch

from haste_b200 import ops

pytestmark = pytest.mark.gpu


def projection(x, W):
    M, H = x.shape[0], W.shape[1]
    z = x.new_zeros
    out = ops.layer_norm_indrnn_forward(False, 0.0, x[None], z(M, H), W, z(H), z(H), x.new_ones(2, H), z(0))
    return out[1][0]


# Errors relative to |x row| |W column|, which is the size of a sum of random signs.  Two planes hold 22
# bits of each operand (2^-23 each, lo.lo dropped: 2^-24); the accumulator truncates 24 times per chunk by
# half a unit of 2^-24 on average, always towards zero: about 12 * 2^-24 + 2 * 2^-23 = 9.5e-7.
BOUND = 1e-6


def relative(got, x, W):
    scale = x.double().norm(dim=1, keepdim=True) * W.double().norm(dim=0, keepdim=True)
    return (got.double() - x.double() @ W.double()).abs() / scale.clamp_min(1e-300)


@pytest.mark.parametrize("M,K,N", [(16384, 512, 1024), (65500, 257, 500), (8193, 1021, 1001), (4099, 2100, 1030),
                                   (130000, 256, 256)])
@pytest.mark.parametrize("spread", [0.0, 3.0])
def test_projection_is_fp32_grade(M, K, N, spread):
    g = torch.Generator("cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=g)
    W = torch.randn(K, N, device="cuda", generator=g) / K ** 0.5
    # rows and columns of very different size, as unnormalised inputs have them
    x *= torch.exp(spread * torch.randn(M, 1, device="cuda", generator=g))
    W *= torch.exp(spread * torch.randn(1, N, device="cuda", generator=g))
    got = projection(x, W)
    for rows in (slice(0, 300), slice(M - 300, M)):
        assert relative(got[rows], x[rows], W).square().mean().sqrt().item() < BOUND


def test_projection_of_extreme_rows_and_columns():
    M, K, N = 16384, 512, 1024
    g = torch.Generator("cuda").manual_seed(1)
    x = torch.randn(M, K, device="cuda", generator=g)
    W = torch.randn(K, N, device="cuda", generator=g) / K ** 0.5
    x[0] = 0.0
    x[1] *= 1e30
    x[2] *= 1e-30
    x[3, 5] = float("inf")
    x[4, 7] = float("nan")
    x[5] *= 1e-3
    x[5, 9] = 1e4
    W[:, 0] = 0.0
    W[:, 1] *= 1e-30
    W[:, 2] *= 1e6
    got = projection(x, W)
    assert (got[0] == 0).all()
    assert not torch.isfinite(got[3]).any()
    assert torch.isnan(got[4]).all()
    assert torch.isfinite(got[8:]).all()
    for r in (1, 2, 5, 6, 7):
        keep = torch.ones(N, dtype=torch.bool, device="cuda")
        keep[1] = r != 2  # 1e-60 is no float
        err = relative(got[r:r + 1], x[r:r + 1], W)[0, keep]
        assert err.square().mean().sqrt().item() < BOUND and err.max().item() < 5 * BOUND, r


@pytest.mark.parametrize("M,K,N", [(16384, 512, 1024), (65536, 300, 500), (4096, 2100, 1030), (8200, 1024, 1024),
                                   (1000, 8200, 1030)])  # the last one: K split
@pytest.mark.parametrize("where", ["row", "column", "nowhere"])
def test_projection_with_values_that_tower_above_their_row(M, K, N, where):
    """A feature of 1e7 among others of 1e-3 that meets a weight of zero, or a weight of 1e7 that meets a feature of zero:
    the result is what the small values make.  Errors relative to the sum of |x| |W|, by the bound above (the
    bf16 planes are handed over as often; a term's own error, 2^-22, is smaller than the accumulator's)."""
    g = torch.Generator("cuda").manual_seed(K)
    x = torch.randn(M, K, device="cuda", generator=g)
    W = torch.randn(K, N, device="cuda", generator=g) / K ** 0.5
    if where == "row":
        x *= 1e-3
        x[M - 7, 3], x[M - 7, K - 1] = 1e7, -1e7
        W[3], W[K - 1] = 0.0, 0.0
    elif where == "column":
        W *= 1e-3
        W[5, N - 3], W[K - 1, N - 3] = 1e7, 3e6
        x[:, 5], x[:, K - 1] = 0.0, 0.0
    got = projection(x, W)
    for rows in (slice(0, 64), slice(M - 64, M)):
        a = x[rows].double()
        err = (got[rows].double() - a @ W.double()).abs() / (a.abs() @ W.double().abs())
        assert err.square().mean().sqrt().item() < BOUND and err.max().item() < 5 * BOUND
        assert err[:, N - 3].max().item() < 5 * BOUND
