"""Prompt attention on tcgen05 around the lines where a launch changes its tile (keys a tile, one query tile or two a block): portions at the edges of
tiles, kept keys, slopes, windows and several page sizes, against the CUDA-core kernel."""
import pytest
import torch

from helpers import scattered_tables

pytestmark = pytest.mark.gpu


def both(rows, H, G, D, page, window=0, keep=0, mods=None, min_q_len=2, work=True, seed=0):
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(seed)
    T, stride = sum(n for n, _ in rows), (H + 2 * G) * D
    n_pages = sum(-(-c // page) for _, c in rows) + 2
    tables = scattered_tables([c for _, c in rows], page, n_pages, seed)
    block = torch.zeros(len(rows), max(len(t) for t in tables), dtype=torch.int32)
    for r, t in enumerate(tables):
        block[r, :len(t)] = torch.tensor(t, dtype=torch.int32)
    k, v = (torch.randn(n_pages, G, page, D, generator=g).bfloat16().cuda() for _ in "kv")
    q = torch.randn(T, stride, generator=g).bfloat16().cuda()
    lens = torch.tensor([n for n, _ in rows], dtype=torch.int32)
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    args = (q, stride, k, v, block.cuda(), starts.cuda(), lens.cuda(), torch.tensor([c for _, c in rows], dtype=torch.int32, device="cuda"), T)
    out = [torch.zeros(T, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    long = [n for n, _ in rows if n >= min_q_len]
    ops.prefill_attention_tc(*args, out[0], H, G, D, page, D ** -0.5, window, min_q_len=min_q_len, work=(len(long), sum(long)) if work else None, mods=mods, keep=keep)
    ops.paged_attention(*args, out[1], H, G, D, page, D ** -0.5, window, min_q_len=min_q_len, mods=mods, keep=keep)
    torch.cuda.synchronize()
    ops.check_tc_errors()
    return out


def close(got, want):
    """Weights and outputs are rounded to bfloat16 (2^-9 each, of values up to the largest output), the reference's once: 1.5e-2 of the largest."""
    assert torch.isfinite(got).all()
    assert (got.float() - want.float()).abs().max() <= 1.5e-2 * max(1.0, want.float().abs().max().item())


# more than 296 blocks: 64 keys a tile with heads of 128; fewer: 128 keys
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows,H,G", [([(1281, 1281)], 32, 8), ([(1152, 1152)], 32, 4), ([(129, 1000), (64, 64), (1, 900), (1100, 1163)], 32, 32), ([(2048, 2048)], 32, 8),
                                      ([(300, 363)], 16, 4), ([(1919, 1919)], 32, 4), ([(128, 128)] * 12, 32, 8), ([(2, 65), (3, 3), (130, 130)], 4, 1)])
def test_launches_of_every_size(rows, H, G, D):
    for page, work in ((16, True), (64, False)):
        close(*both(rows, H, G, D, page, work=work))


@pytest.mark.parametrize("window,keep", [(100, 0), (-96, 0), (200, 40), (64, 200), (1, 0)])
@pytest.mark.parametrize("rows", [[(1500, 1500)], [(700, 900), (650, 650)]])
def test_windows_and_kept_keys_with_64_keys_a_tile(rows, window, keep):
    close(*both(rows, 32, 4, 128, 16, window=window, keep=keep))


@pytest.mark.parametrize("page", [8, 32, 128])
def test_pages_with_64_keys_a_tile(page):
    close(*both([(1300, 1400), (70, 70)], 32, 8, 128, page))


@pytest.mark.parametrize("what", ["slope", "cap", "bias", "sink"])
def test_modified_scores_in_large_launches(what):
    from mini_inference_engine_b200.kernels import ops
    H = 32
    g = torch.Generator().manual_seed(1)
    mods = ops.ScoreMods(3.0 if what == "cap" else 0.0, torch.randn(H, generator=g).cuda() if what == "sink" else None,
                         torch.randn(H, 90, generator=g).cuda() if what == "bias" else None, (torch.rand(H, generator=g) * 0.1).cuda() if what == "slope" else None)
    close(*both([(1400, 1500)], H, 8, 128, 16, mods=mods))


@pytest.mark.parametrize("n", [300, 800, 1500])
def test_fewer_keys_a_tile_lose_no_precision(n):
    """The same heads in a launch of few blocks (128 keys a tile) and, each twice, in one of many (64 keys): the error against 64 bits is no larger.  (Over some 30,000 rows,
    whose squared errors scatter by one and a half times their mean, the two norms differ by about half a percent by chance: four times that is allowed.  With the
    sums of unrounded weights the smaller tiles' error is 5 to 8 percent larger.)"""
    from mini_inference_engine_b200.kernels import ops
    G, D, page = 288 // -(-n // 128), 128, 16
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    pages = -(-n // page)
    k, v, q = rnd(pages, G, page, D).bfloat16(), rnd(pages, G, page, D).bfloat16(), (rnd(n, G, D) * 1.5).bfloat16()
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device="cuda")
    table = torch.arange(pages, dtype=torch.int32, device="cuda").view(1, -1)
    flat = lambda t: t.permute(1, 0, 2, 3).reshape(G, -1, D)[:, :n].double()
    scores = q.double().permute(1, 0, 2) @ flat(k).transpose(1, 2) * D ** -0.5
    scores = scores.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), -float("inf"))
    want = (torch.softmax(scores, -1) @ flat(v)).permute(1, 0, 2)
    errors = []
    for times in (1, 2):
        H = G * times
        qs = q.repeat_interleave(times, 1).reshape(n, H * D).contiguous()
        out = torch.empty(n, H, D, device="cuda")
        ops.prefill_attention_tc(qs, H * D, k, v, table, i32(0), i32(n), i32(n), n, out, H, G, D, page, D ** -0.5, 0, work=(1, n))
        torch.cuda.synchronize()
        ops.check_tc_errors()
        errors.append((out.view(n, G, times, D)[:, :, 0].double() - want).norm().item())
    print(f"{n} tokens: {errors[1] / errors[0] - 1:+.2%}")
    assert errors[1] <= 1.02 * errors[0]


@pytest.mark.parametrize("D", [64, 128])
def test_more_rows_than_a_grid_is_high(D):
    """70,000 portions of two tokens in a step (a tile each) against the CUDA-core kernel."""
    from mini_inference_engine_b200.kernels import ops
    rows, page = 70000, 8
    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    k, v, q = rnd(rows + 1, 1, page, D), rnd(rows + 1, 1, page, D), rnd(2 * rows, 2 * D)
    i32 = dict(dtype=torch.int32, device="cuda")
    args = (q, 2 * D, k, v, torch.randperm(rows, device="cuda").int().add(1).view(rows, 1), torch.arange(0, 2 * rows, 2, **i32), torch.full((rows,), 2, **i32),
            torch.full((rows,), 5, **i32), 2 * rows)
    out = [torch.zeros(2 * rows, 2, D, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    ops.prefill_attention_tc(*args, out[0], 2, 1, D, page, D ** -0.5, 0, work=(rows, 2 * rows))
    ops.paged_attention(*args, out[1], 2, 1, D, page, D ** -0.5, 0)
    torch.cuda.synchronize()
    ops.check_tc_errors()
    close(*out)
