"""Float32 attention of prompt portions in tiles of 64 (token, head) pairs against the kernel that gives a warp one pair, over masks, kept keys,
score modifiers, group sizes, head sizes and page sizes."""
import pytest
import torch

from helpers import scattered_tables

pytestmark = pytest.mark.gpu

ROWS = [(64, 64), (1, 70), (9, 9), (130, 200), (2, 3), (33, 400), (65, 65)]


def case(rows, H, G, D, page, seed=0):
    g = torch.Generator().manual_seed(seed)
    T, stride = sum(n for n, _ in rows), (H + 2 * G) * D
    n_pages = sum(-(-c // page) for _, c in rows) + 2
    tables = scattered_tables([c for _, c in rows], page, n_pages, seed)
    block = torch.zeros(len(rows), max(len(t) for t in tables), dtype=torch.int32)
    for r, t in enumerate(tables):
        block[r, :len(t)] = torch.tensor(t, dtype=torch.int32)
    k, v = (torch.randn(n_pages, G, page, D, generator=g).cuda() for _ in "kv")
    q = torch.randn(T, stride, generator=g).cuda()
    lens = torch.tensor([n for n, _ in rows], dtype=torch.int32)
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    args = (q, stride, k, v, block.cuda(), starts.cuda(), lens.cuda(), torch.tensor([c for _, c in rows], dtype=torch.int32, device="cuda"), T)
    return args, tables, torch.zeros(T, H, D, device="cuda")


def both(args, out, H, G, D, page, min_q_len=1, **how):
    from mini_inference_engine_b200.kernels import ops
    window = how.pop("window", 0)
    a = ops.attention_f32(*args, out.clone(), H, G, D, page, D ** -0.5, window, min_q_len=min_q_len, **how)
    b = ops.paged_attention(*args, out.clone(), H, G, D, page, D ** -0.5, window, min_q_len=min_q_len, **how)
    torch.cuda.synchronize()
    ops.check_range_errors()
    return a, b


def close(a, b, v):
    """Scores of a few units differ by about sqrt(D) 2^-24 of sum |q||k| between the two orders of summation, some 3e-6, weights by as much of
    themselves, outputs by as much of the largest value: 1e-5 of it leaves three times that."""
    assert torch.isfinite(a).all()
    assert (a - b).abs().max().item() <= 1e-5 * v.abs().max().item()


@pytest.mark.parametrize("H,G,D", [(8, 1, 64), (4, 4, 32), (6, 2, 48), (32, 4, 64), (14, 2, 80), (4, 1, 128), (10, 1, 16), (3, 3, 112)])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 0), (-64, 0), (50, 20), (70, 130), (-48, 10)])
def test_masks_groups_and_head_sizes(H, G, D, window, keep):
    args, _, out = case(ROWS, H, G, D, 16, H + D)
    close(*both(args, out, H, G, D, 16, window=window, keep=keep), args[3])


@pytest.mark.parametrize("page", [1, 8, 64, 128])
def test_page_sizes(page):
    args, _, out = case(ROWS, 8, 2, 64, page, page)
    close(*both(args, out, 8, 2, 64, page, window=33, keep=5), args[3])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("what", ["cap", "sink", "bias", "slope", "all"])
def test_score_modifiers(what, D):
    from mini_inference_engine_b200.kernels import ops
    H, G = 8, 2
    g = torch.Generator().manual_seed(3)
    on = lambda n: what in (n, "all")
    mods = ops.ScoreMods(2.0 if on("cap") else 0.0, torch.randn(H, generator=g).cuda() if on("sink") else None,
                         torch.randn(H, 50, generator=g).cuda() if on("bias") else None, torch.rand(H, generator=g).cuda() if on("slope") else None)
    args, _, out = case(ROWS, H, G, D, 16)
    close(*both(args, out, H, G, D, 16, mods=mods), args[3])
    close(*both(args, out, H, G, D, 16, mods=mods, window=37, keep=9), args[3])


def test_short_rows_are_left_alone_by_one_and_long_rows_by_the_other():
    from mini_inference_engine_b200.kernels import ops
    H, G, D = 8, 2, 64
    args, _, out = case(ROWS, H, G, D, 16)
    whole = ops.paged_attention(*args, out.clone(), H, G, D, 16, D ** -0.5)
    work = (sum(n >= 9 for n, _ in ROWS), sum(n for n, _ in ROWS if n >= 9))
    for hint in (None, work):
        got = torch.full_like(out, 7.0)
        ops.attention_f32(*args, got, H, G, D, 16, D ** -0.5, min_q_len=9, work=hint)
        at = 0
        for n, _ in ROWS:
            assert bool((got[at:at + n] == 7.0).all()) == (n < 9)
            at += n
        ops.paged_attention(*args, got, H, G, D, 16, D ** -0.5, below=9)
        close(got, whole, args[3])


def test_a_value_that_is_not_finite_reaches_only_the_queries_that_see_it():
    """The key and value of one position, in a tile that earlier queries' blocks also load."""
    H, G, D, page = 8, 2, 64, 16
    args, tables, out = case([(100, 100)], H, G, D, page)
    for cache, bad in ((args[3], float("inf")), (args[2], float("nan"))):
        cache[tables[0][70 // page], :, 70 % page] = bad
    a, b = both(args, out, H, G, D, page)
    assert torch.isfinite(a[:70]).all() and torch.equal(torch.isfinite(a), torch.isfinite(b))
    close(a[:70], b[:70], torch.ones(1, device="cuda"))


def test_the_step_takes_it_in_float32():
    from types import SimpleNamespace
    from mini_inference_engine_b200.kernels import attention, ops
    H, G, D, page = 8, 2, 64, 16
    args, _, out = case(ROWS, H, G, D, page)
    q, stride, k, v, block, starts, lens, ctx_lens, T = args
    cache = SimpleNamespace(k=k, v=v, group=0, page_size=page)
    want = ops.paged_attention(*args, out.clone(), H, G, D, page, D ** -0.5)
    for host in ({"q_len": [n for n, _ in ROWS]}, {"q_len": None}):           # the second: a captured step
        ctx = SimpleNamespace(block_tables=[block], row_q_start=starts, row_q_len=lens, row_ctx_len=ctx_lens, num_tokens=T, max_ctx_len=400, host=host)
        got = attention.attention(q, ctx, cache, torch.zeros_like(out), H, G, D, D ** -0.5, 0)
        close(got, want, v)


@pytest.mark.parametrize("rows,max_ctx,host,kernels", [([(40, 600)], 600, True, {"paged"}), ([(200, 600)], 600, True, {"tiles"}), ([(200, 600), (1, 50)], 600, True, {"paged", "tiles"}),
                                                       ([(200, 200)], 200, True, {"paged"}), ([(256, 256)], 256, True, {"tiles"}), ([(150, 600)], 600, False, {"paged"}),
                                                       ([(250, 600)], 600, False, {"paged", "tiles"}), ([(1, 90)] * 300, 90, True, {"paged"})])
def test_a_step_of_few_pairs_is_left_to_the_warps(monkeypatch, rows, max_ctx, host, kernels):
    """Eight heads: 192 tokens are enough beside earlier positions, 256 without."""
    from types import SimpleNamespace
    from mini_inference_engine_b200.kernels import attention, ops
    H, G, D, page = 8, 2, 64, 16
    args, _, out = case(rows, H, G, D, page)
    q, stride, k, v, block, starts, lens, ctx_lens, T = args
    want = ops.paged_attention(*args, out.clone(), H, G, D, page, D ** -0.5)
    used, paged, tiles = set(), ops.paged_attention, ops.attention_f32
    monkeypatch.setattr(ops, "paged_attention", lambda *a, **h: (used.add("paged"), paged(*a, **h))[1])
    monkeypatch.setattr(ops, "attention_f32", lambda *a, **h: (used.add("tiles"), tiles(*a, **h))[1])
    ctx = SimpleNamespace(block_tables=[block], row_q_start=starts, row_q_len=lens, row_ctx_len=ctx_lens, num_tokens=T, max_ctx_len=max_ctx,
                          host={"q_len": [n for n, _ in rows] if host else None})
    got = attention.attention(q, ctx, SimpleNamespace(k=k, v=v, group=0, page_size=page), torch.zeros_like(out), H, G, D, D ** -0.5, 0)
    close(got, want, v)
    assert used == kernels


@pytest.mark.parametrize("what", ["page", "context"])
def test_a_number_out_of_range_is_reported_under_this_kernel_s_name(what):
    """A page that is not in the pool (page 0 is read in its place), and more positions than the block table covers (the row is left alone)."""
    from mini_inference_engine_b200.kernels import ops
    H, G, D, page = 8, 2, 64, 16
    args, _, out = case([(70, 70)], H, G, D, page)
    args = list(args)
    if what == "page":
        args[4][0, 1] = args[2].shape[0]
    else:
        args[7] = args[7] + 1000
    ops.check_range_errors()
    ops.attention_f32(*args, out, H, G, D, page, D ** -0.5, 0)
    torch.cuda.synchronize()
    with pytest.raises(ops.KernelError, match="attention_f32"):
        ops.check_range_errors()
