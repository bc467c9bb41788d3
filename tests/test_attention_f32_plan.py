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
        assert shares in (1, 2, 4, 8) and shares <= max(1, 2 * -(-max_ctx // 64))
        # what a B200 runs at once in clusters of four and eight (a block of eight warps over heads of 128 has an SM to itself, of four over heads of 64 a third)
        places = {4: 132, 8: 120} if head_dim == 128 else {4: 416, 8: 384}
        assert shares <= 2 or shares * items <= places[shares], (rows, tokens, warps, shares)


def test_decoding_rows_and_portions_of_heads_of_128():
    # 32 heads on 8: 1, 4, 8 rows of one token on up to 960 positions; one row of 32 and of 100 tokens
    assert [plan(r * 4, r, 32, 8, 128, 960)[:2] for r in (1, 4, 8)] == [(8, 8), (8, 4), (8, 2)]
    assert [plan(n * 4, 1, 32, 8, 128, 2048)[:2] for n in (32, 100)] == [(8, 8), (8, 4)]
