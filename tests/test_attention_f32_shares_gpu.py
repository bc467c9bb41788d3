"""Float32 attention by tiles where a walk of keys is shared out over the blocks of a cluster, in blocks of eight warps, for rows of one token, and for numbers that have no
three bfloat16 parts -- against the kernel that gives a warp one pair."""
from types import SimpleNamespace

import pytest
import torch

from test_attention_f32_gpu import both, case, close

pytestmark = pytest.mark.gpu

LONG = [(3, 1200), (1, 1100), (17, 700), (1, 5), (64, 64), (2, 513)]


@pytest.mark.parametrize("H,G,D", [(16, 2, 64), (4, 4, 48), (8, 2, 128), (3, 1, 96), (20, 20, 80)])
@pytest.mark.parametrize("window,keep", [(0, 0), (300, 0), (-256, 70)])
@pytest.mark.parametrize("max_ctx", [None, 64, 1200])
def test_walks_in_one_to_eight_shares(H, G, D, window, keep, max_ctx):
    """``max_ctx`` only shapes the launch: too small a number is slow, not wrong."""
    args, _, out = case(LONG, H, G, D, 16, H + D)
    from mini_inference_engine_b200.kernels import ops
    a = ops.attention_f32(*args, out.clone(), H, G, D, 16, D ** -0.5, window, keep=keep, max_ctx=max_ctx)
    b = ops.paged_attention(*args, out.clone(), H, G, D, 16, D ** -0.5, window, keep=keep)
    torch.cuda.synchronize()
    ops.check_range_errors()
    close(a, b, args[3])


@pytest.mark.parametrize("rows", [[(640, 700)], [(400, 900), (350, 350), (1, 1000)]])
@pytest.mark.parametrize("sink", [False, True])
def test_wide_blocks(rows, sink):
    from mini_inference_engine_b200.kernels import ops
    H, G, D = 32, 4, 64
    mods = ops.ScoreMods(0.0, torch.linspace(-2.0, 3.0, H).cuda(), None, None) if sink else None
    args, _, out = case(rows, H, G, D, 16)
    close(*both(args, out, H, G, D, 16, mods=mods), args[3])


@pytest.mark.parametrize("H,G,D", [(8, 2, 64), (8, 2, 128), (10, 10, 128)])          # (the last: blocks of four warps without memory for keys on their way)
@pytest.mark.parametrize("what", ["key", "value", "query"])
@pytest.mark.parametrize("bad", [3e38, float("inf"), float("nan")])
def test_numbers_without_parts_reach_what_they_reach_one_by_one(H, G, D, what, bad):
    """One number of one position, or of one query; whole tiles are multiplied number by number then."""
    rows, page = [(300, 700), (5, 700)], 16
    args, tables, out = case(rows, H, G, D, page)
    at = 640
    if what == "query":
        args[0][at - 400, 3 * D + 5] = bad                     # the row's first token is at position 400
    else:
        args[2 if what == "key" else 3][tables[0][at // page], 1, at % page, 7] = bad
    a, b = both(args, out, H, G, D, page)
    assert torch.isfinite(a[:at - 400]).all() and torch.isfinite(a[300:]).all() and torch.equal(torch.isfinite(a), torch.isfinite(b))
    ok = torch.isfinite(b) & (b.abs() < 1e6)
    assert ((a - b).abs()[ok] <= 2e-5 * b[ok].abs().max()).all()
    big = torch.isfinite(b) & (b.abs() >= 1e6)
    assert ((a - b).abs()[big] <= 1e-4 * b.abs()[big]).all()


@pytest.mark.parametrize("H,G,D,rows,ctx,kernels", [(8, 1, 64, [(1, 128)] * 70, 128, {"tiles"}), (8, 1, 64, [(1, 127)] * 3, 127, {"paged"}), (4, 4, 64, [(1, 300)] * 16, 300, {"tiles"}),
                                                    (4, 4, 64, [(1, 300)] * 17, 300, {"paged"}), (16, 2, 128, [(1, 300)] * 33, 300, {"paged"}),
                                                    (8, 1, 64, [(2, 640), (1, 30)], 640, {"tiles"}), (4, 4, 64, [(20, 640)] + [(1, 30)] * 17, 640, {"tiles", "paged"}),
                                                    (4, 4, 64, [(20, 70)] + [(1, 640)] * 17, 640, {"paged"}), (4, 4, 64, [(9, 640)] + [(1, 30)] * 17, 640, {"paged"}), (8, 1, 64, [(2, 639), (1, 30)], 639, {"paged"}),
                                                    (32, 8, 128, [(64, 64)], 64, {"paged"}), (32, 8, 128, [(64, 64)] * 2, 64, {"tiles"}), (16, 16, 96, [(20, 20)] * 32, 20, {"paged"}),
                                                    (16, 16, 96, [(40, 40)] * 16, 40, {"tiles"}), (32, 8, 128, [(64, 64)] * 2 + [(1, 90)] * 9, 90, {"tiles", "paged"})])
def test_rows_of_one_token_and_long_rows_of_few(monkeypatch, H, G, D, rows, ctx, kernels):
    from mini_inference_engine_b200.kernels import attention, ops
    args, _, out = case(rows, H, G, D, 16)
    q, stride, k, v, block, starts, lens, ctx_lens, T = args
    want = ops.paged_attention(*args, out.clone(), H, G, D, 16, D ** -0.5)
    used, paged, tiles = set(), ops.paged_attention, ops.attention_f32
    monkeypatch.setattr(ops, "paged_attention", lambda *a, **h: (used.add("paged"), paged(*a, **h))[1])
    monkeypatch.setattr(ops, "attention_f32", lambda *a, **h: (used.add("tiles"), tiles(*a, **h))[1])
    step = SimpleNamespace(block_tables=[block], row_q_start=starts, row_q_len=lens, row_ctx_len=ctx_lens, num_tokens=T, max_ctx_len=ctx,
                           host={"q_len": [n for n, _ in rows], "ctx_len": [c for _, c in rows]})
    got = attention.attention(q, step, SimpleNamespace(k=k, v=v, group=0, page_size=16), torch.zeros_like(out), H, G, D, D ** -0.5, 0)
    close(got, want, v)
    assert used == kernels


@pytest.mark.parametrize("window,keep", [(0, 0), (300, 0), (-256, 70)])
@pytest.mark.parametrize("what", ["key", "value", "query"])
@pytest.mark.parametrize("bad", [3e38, float("inf"), float("nan")])
def test_numbers_without_parts_in_wide_blocks(window, keep, what, bad):
    """Blocks of eight warps (32 heads on 4, 640 tokens): a number in an early tile, while the next tile's keys are on their way."""
    H, G, D, page, at = 32, 4, 64, 16, 130
    args, tables, out = case([(640, 700)], H, G, D, page)
    if what == "query":
        args[0][at - 60, 3 * D + 5] = bad                      # the row's first token is at position 60
    else:
        args[2 if what == "key" else 3][tables[0][at // page], 1, at % page, 7] = bad
    a, b = both(args, out, H, G, D, page, window=window, keep=keep)
    again, _ = both(args, out, H, G, D, page, window=window, keep=keep)
    assert torch.equal(a.view(torch.int32), again.view(torch.int32))
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(a), kind(b))
    ok = torch.isfinite(b) & (b.abs() < 1e6)
    assert ok.float().mean() > 0.5 and ((a - b).abs()[ok] <= 2e-5 * b[ok].abs().max()).all()
    big = torch.isfinite(b) & (b.abs() >= 1e6)
    assert ((a - b).abs()[big] <= 1e-4 * b.abs()[big]).all()


@pytest.mark.parametrize("H,G,D", [(8, 2, 64), (8, 2, 128), (10, 10, 128)])          # (the last: blocks of four warps without memory for keys on their way)
@pytest.mark.parametrize("n,ctx,first,end", [(100, 100, 64, 65), (150, 150, 128, 129), (1, 129, 128, 129), (1, 129, 64, 129), (300, 520, 192, 256), (300, 520, 0, 64), (300, 520, 0, 448),
                                             (300, 520, 64, 520), (5, 700, 0, 700)])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("window,keep", [(0, 0), (150, 0), (-128, 70)])
def test_shares_of_scores_that_are_no_numbers(H, G, D, n, ctx, first, end, sink, window, keep):
    """Keys that are NaN from position ``first`` up to ``end``: whatever share of a walk meets them, the outputs are no numbers where the walk in one share has none."""
    from mini_inference_engine_b200.kernels import ops
    args, tables, out = case([(n, ctx), (70, 700)], H, G, D, 16)
    for at in range(first, end):
        args[2][tables[0][at // 16], 1, at % 16] = float("nan")
    mods = ops.ScoreMods(0.0, torch.linspace(-2.0, 3.0, H).cuda(), None, None) if sink else None
    res = [ops.attention_f32(*args, out.clone(), H, G, D, 16, D ** -0.5, window, keep=keep, mods=mods, max_ctx=c) for c in (64, 128, 200, 700, 1 << 20)]
    warps = ops.paged_attention(*args, out.clone(), H, G, D, 16, D ** -0.5, window, keep=keep, mods=mods)
    torch.cuda.synchronize()
    for a in res[1:]:
        assert torch.equal(torch.isnan(a), torch.isnan(res[0]))
        ok = ~torch.isnan(a)
        assert ((a - res[0]).abs()[ok] <= 2e-5 * args[3].abs().max()).all()
    heads = slice(0, H // G)
    assert torch.isfinite(res[0][:, heads]).all() and torch.isfinite(res[0][n:]).all()        # (the other key head, the other row)
    if first % 64:                                             # (a tile of 64 keys that are all NaN counts as out of sight in front of the first number; the other kernel's are 32)
        return
    if end - first <= 64 and first > 0 and not window:
        assert torch.equal(torch.isnan(warps), torch.isnan(res[0]))
