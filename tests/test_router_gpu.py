"""The router's product and choice in one launch at the edges of their steps: an odd number of outputs, column segments that the rounding leaves empty, rows without
16-byte pieces, one to eight tokens a block and a last block with fewer, choices of one to more than a warp's lanes, logits that tie or are not numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("E,top", [(1, 1), (5, 2), (16, 4), (33, 32), (64, 8), (70, 33), (260, 6)])
@pytest.mark.parametrize("h", [40, 1002, 1100, 2048])
@pytest.mark.parametrize("T", [1, 300, 603, 1184, 1201])
def test_router_against_the_product_and_the_choice_by_one_thread(E, top, h, T):
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(E * h + T)
    x = torch.randn(T, h, generator=g, device=DEV).bfloat16()
    w = torch.randn(E, h, generator=g, device=DEV)
    if E > 4:
        w[3] = w[1]                                            # two outputs that tie
    if T > 1:
        x[T // 2, 1] = float("nan")
    for dt in (torch.bfloat16, torch.float32):
        for score, real in (("top_softmax", None), ("sigmoid", None), ("top_softmax", max(1, E - 2)), ("sigmoid", max(1, E - 2))):
            rule = ops.RouteRule(score, real=real)
            logits = torch.empty(T, E, device=DEV)
            got = ops.moe_router(x.to(dt), w, top, logits, rule)
            want = ops.moe_route(logits, top, rule)
            assert len(got) == len(want)
            assert torch.equal(got[0], want[0])
            for a, b in zip(got[1:], want[1:]):                # the same operations in the same order: the same bits
                assert torch.equal(a.nan_to_num(-7.0), b.nan_to_num(-7.0))
            fine = torch.ones(T, dtype=torch.bool, device=DEV)
            if T > 1:
                fine[T // 2] = False
            wide = x.double() @ w.double().t()
            limit = 2.0 ** -24 * (h / 32 + 16) * (x.double().abs() @ w.double().abs().t())      # a lane's chain of h / 32 terms, then the sums over lanes and segments
            assert ((logits.double() - wide).abs()[fine] <= limit[fine]).all()
