"""Linear attention with decays in chunks as matrix products against the token-by-token kernel, over head sizes, row lengths at the edges of
chunks, decays per head and per token, activations, the column of ones, types and a step whose row lengths the host does not know."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [1, 65, 64, 128, 3, 129, 200, 63, 640]


def scan(monkeypatch, chunked, rows, H, D, V, dt, *, per_token=False, act=False, ones=False, rot=0, known=True, seed=0, spoil=None):
    from mini_inference_engine_b200.kernels import ops
    monkeypatch.setattr(ops, "decay_chunks_take", (lambda d: d % 4 == 0 and d <= 128) if chunked else (lambda d: False))
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, dv = sum(rows), V + int(ones)
    qkv = rnd(T, H * (2 * D + V) + 8).to(dt)
    state = rnd(len(rows) + 1, H, dv, D)
    lens = torch.tensor(rows, dtype=torch.int32, device="cuda")
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    slots = torch.tensor([len(rows) - i for i in range(len(rows))], dtype=torch.int32, device="cuda")
    pos = torch.cat([torch.arange(n, dtype=torch.int32) + 7 * i for i, n in enumerate(rows)]).cuda()
    how = dict(decay=torch.rand(H, generator=g, device="cuda") * 0.2 + 0.8)
    if per_token:
        keep = torch.rand(T, H, generator=g, device="cuda")
        keep[5::17], keep[9::23] = 0.0, 1.0
        how = dict(tok_decay=keep, k_tok=torch.rand(T, H, generator=g, device="cuda"))
    if spoil is not None:
        qkv[spoil] = float("inf")
    out = torch.zeros(T, H * dv, device="cuda")
    freq = torch.rand(rot // 2, generator=g, device="cuda") if rot else None
    ops.decay_scan(qkv, pos, starts, lens, slots, state, out, num_heads=H, dim=D, vdim=V, max_q_len=max(rows), act=act, ones=ones, q_scale=0.5, k_scale=D ** -0.5,
                   freq=freq, rot=rot, q_lens=rows if known else None, **how)
    torch.cuda.synchronize()
    return out, state


def close(got, want):
    """Both sum in float32, up to some hundred terms that matter (decays of 0.8 to 1) in different orders: 2^-24 sqrt(several hundred) of the
    largest result, ten times over."""
    for a, b in zip(got, want):
        assert torch.isfinite(a).all()
        assert (a - b).abs().max().item() <= 1.5e-5 * b.abs().max().item()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V", [(2, 128, 256), (3, 64, 64), (1, 20, 33), (2, 100, 130), (5, 4, 3), (2, 68, 65)])
@pytest.mark.parametrize("per_token,act,ones,rot", [(False, False, False, 0), (False, True, False, 0), (True, False, True, 0), (False, False, False, -1), (True, True, False, 0)])
def test_chunks_against_tokens(monkeypatch, dt, H, D, V, per_token, act, ones, rot):
    how = dict(per_token=per_token, act=act, ones=ones, rot=D // 2 // 2 * 2 if rot else 0, seed=H + D + V)
    close(scan(monkeypatch, True, ROWS, H, D, V, dt, **how), scan(monkeypatch, False, ROWS, H, D, V, dt, **how))


@pytest.mark.parametrize("rows", [[65], [300, 100], [64, 10, 1], [1, 1, 90], [4096]])
@pytest.mark.parametrize("known", [True, False])
def test_rows_the_host_knows_or_not(monkeypatch, rows, known):
    close(scan(monkeypatch, True, rows, 2, 32, 40, torch.float32, known=known, ones=True, per_token=True),
          scan(monkeypatch, False, rows, 2, 32, 40, torch.float32, ones=True, per_token=True))


def test_a_token_that_is_not_finite_spoils_only_what_follows(monkeypatch):
    out, state = scan(monkeypatch, True, [150, 70], 2, 32, 40, torch.float32, spoil=100)
    ref, ref_state = scan(monkeypatch, False, [150, 70], 2, 32, 40, torch.float32, spoil=100)
    assert torch.isfinite(out[:100]).all() and torch.isfinite(out[150:]).all()
    assert torch.equal(torch.isfinite(out), torch.isfinite(ref)) and torch.equal(torch.isfinite(state), torch.isfinite(ref_state))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_preparation_of_rows_that_start_anywhere(monkeypatch, dt):
    """Sizes and starts that do not allow four entries at a time give what those that do give."""
    from mini_inference_engine_b200.kernels import ops
    H, D, V, T, rot = 3, 24, 16, 40, 16
    g = torch.Generator(device="cuda").manual_seed(1)
    wide = torch.randn(T, H * (2 * D + V) + 4, generator=g, device="cuda").to(dt)
    odd = torch.empty(T * (wide.shape[1] + 1) + 1, dtype=dt, device="cuda")[1:].view(T, -1)[:, :wide.shape[1]].copy_(wide)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    res = []
    for rows in (wide, odd):
        state, out = torch.zeros(2, H, V, D, device="cuda"), torch.zeros(T, H * V, device="cuda")
        ops.retention_scan(rows, torch.arange(T, dtype=torch.int32, device="cuda"), i32(0), i32(T), i32(1), torch.full((H,), 0.9, device="cuda"),
                           torch.rand(rot // 2, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda"), state, out, num_heads=H, dim=D, vdim=V,
                           rot=rot, k_scale=0.2, max_q_len=T)
        res.append((out, state))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("heads", [1, 2, 3])
def test_some_heads_at_a_time(monkeypatch, heads, known):
    """Scratch memory for that many heads at a time: every number as with all at once."""
    from mini_inference_engine_b200.kernels import ops
    for how in (dict(per_token=True, ones=True), dict(act=True)):
        whole = scan(monkeypatch, True, ROWS, 5, 68, 70, torch.bfloat16, known=known, **how)
        with monkeypatch.context() as m:
            m.setattr(ops, "_heads_a_pass", lambda all_heads, bytes_a_head: heads)
            got = scan(m, True, ROWS, 5, 68, 70, torch.bfloat16, known=known, **how)
        assert all(torch.equal(a, b) for a, b in zip(got, whole))
