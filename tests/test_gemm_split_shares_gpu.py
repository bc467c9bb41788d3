"""The float32 product on the tensor cores where the first tiles take all of K and the rest shares of it: every tile width and number of tiles in front, outputs that are not
finite on either side of the line, and sizes whose plan has both."""
import pytest
import torch

from test_gemm_split_gpu import check, operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("splits,whole", [(2, 1), (3, 2), (8, 1)])
@pytest.mark.parametrize("M,N", [(9, 513), (300, 700), (260, 768)])
def test_every_tile_with_shares_behind(bn, splits, whole, M, N):
    from mini_inference_engine_b200.kernels import gemm_split, gemm_tc, ops
    x, w, bias = operands(M, N, 64 * 11 + 5, bn + whole)
    for b in (bias, None):
        check(gemm_split.gemm_split(x, w, torch.empty(M, N, device="cuda"), b, force=(bn, splits, whole)), x, w, b)
    w[3, 5], w[N - 1, 700], x[4, 9], x[M - 1, 30] = float("inf"), float("nan"), -float("inf"), 1e-40
    got = gemm_split.gemm_split(x, w, torch.empty(M, N, device="cuda"), bias, force=(bn, splits, whole))
    want = ops.gemm_simt(x, w, torch.empty(M, N, device="cuda"), bias)
    torch.cuda.synchronize()
    gemm_tc.check_error()
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(want))
    fine = torch.isfinite(want)
    room = 8 * x.shape[1] ** 0.5 * 2.0 ** -24 * (x.abs() @ w.abs().t() + bias.abs())           # both sides' distance from the true sums
    assert ((got - want).abs() <= room)[fine].all()


@pytest.mark.parametrize("M,N,K", [(1000, 2560, 2048), (509, 5632, 1024), (400, 11264, 512)])
def test_sizes_whose_plan_has_both(M, N, K):
    from mini_inference_engine_b200.kernels import gemm_split
    assert gemm_split.plan(M, N, K)[2] > 0
    x, w, bias = operands(M, N, K, 1)
    out = gemm_split.gemm_split(x, w, torch.empty(M, N, device="cuda"), bias)
    check(out, x, w, bias)
    off = lambda t: ((t.double() - (x.double() @ w.double().t() + bias.double())).norm() / t.double().norm()).item()
    # as far from 64 bits as one chain of chunks (measured 0.98 to 0.99 times as far: a share's sums are shorter)
    assert off(out) <= 1.05 * off(gemm_split.gemm_split(x, w, torch.empty_like(out), bias, force=(128, 1)))
