"""The launch plan of float32 attention's tiles, on the host: items for every tile that a step's rows can have, and shares of a walk against the places that the SMs have for blocks."""
import ctypes
import random

import pytest

from mini_inference_engine_b200.kernels import build


def plan(pairs, rows, heads, kv_heads, head_dim, max_ctx, window=0, keep=0, sms=148):
    fn = build.load("attention_f32").mie_attention_f32_plan
    fn.restype = ctypes.c_longlong
    got = fn(ctypes.c_longlong(pairs), rows, heads, kv_heads, head_dim, window, keep, max_ctx, sms)
    return got % 16, got // 16 % 16, got // 256


@pytest.mark.parametrize("group", [1, 2, 3, 4, 6, 8, 12, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_items_for_every_tile(group, head_dim):
    rng = random.Random(group)
    for _ in range(300):
        rows = [rng.choice([1, 1, 2, 5, 16, 33, 64, 127, 700]) for _ in range(rng.randint(1, 20))]
        warps, _, items = plan(sum(rows) * group, len(rows), 2 * group, 2, head_dim, rng.choice([64, 512, 4096]))
        assert items >= 2 * sum(-(-n * group // (16 * warps)) for n in rows)
        assert len(rows) > 1 or items <= 2 * -(-rows[0] * group // (16 * warps))            # (one row: no more than that)


@pytest.mark.parametrize("group", [1, 4, 8])
@pytest.mark.parametrize("kv_heads", [1, 4, 8, 16])
@pytest.mark.parametrize("max_ctx", [64, 128, 200, 960, 4096])
@pytest.mark.parametrize("head_dim", [64, 128])
def test_more_than_two_shares_fit_beside_one_another(group, kv_heads, max_ctx, head_dim):
    for rows, tokens in [(1, 1), (4, 4), (8, 8), (16, 16), (64, 64), (1, 47), (1, 100), (2, 300), (1, 2000)]:
        warps, shares, items = plan(tokens * group, rows, group * kv_heads, kv_heads, head_dim, max_ctx)
        assert shares in (1, 2, 4, 8) and (max_ctx > 64 or shares == 1) and shares <= 2 * -(-max_ctx // 64)
        # what a B200 runs at once in clusters of four and eight: blocks of four warps over heads of 64 have a third of an SM
        if head_dim == 64:
            assert shares <= 2 or shares * items <= {4: 416, 8: 384}[shares], (rows, tokens, warps, shares)


@pytest.mark.parametrize("rows,tokens,ctx,heads,kv_heads,best", [
    (1, 64, 64, 32, 8, (8, 1)), (8, 40, 40, 32, 8, (8, 1)), (32, 20, 20, 16, 2, (8, 1)), (4, 100, 100, 32, 8, (8, 1)), (4, 100, 400, 32, 8, (8, 1)), (1, 100, 230, 32, 8, (8, 4)),
    (2, 64, 364, 32, 8, (8, 4)), (2, 64, 1064, 32, 8, (8, 4)), (1, 500, 800, 32, 8, (8, 2)), (32, 40, 40, 16, 16, (4, 1)), (32, 64, 194, 16, 16, (4, 1)), (16, 64, 64, 16, 16, (4, 1)),
    (16, 1, 400, 32, 8, (4, 2)), (8, 1, 400, 32, 8, (4, 4)), (16, 1, 400, 16, 16, (4, 1))])
def test_heads_of_128_by_the_plan_that_took_least(rows, tokens, ctx, heads, kv_heads, best):
    """As measured on a B200 by every width and number of shares."""
    assert plan(rows * tokens * heads // kv_heads, rows, heads, kv_heads, 128, ctx)[:2] == best
