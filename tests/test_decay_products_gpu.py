"""The chunked decay recurrence's products as bfloat16 parts: shares of the value columns and narrow blocks of few chunks, whole blocks of many, values that are one part or
three, values without parts, and how far the results are from 64 bits."""
import pytest
import torch

from test_decay_chunks_gpu import close, scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,H", [([66], 1), ([128, 70], 3), ([640], 8), ([1000, 900], 6), ([2000], 12)])
@pytest.mark.parametrize("D,V", [(128, 300), (64, 64), (96, 129), (32, 5)])
def test_shares_and_blocks_of_every_size(monkeypatch, dt, rows, H, D, V):
    how = dict(per_token=True, ones=V % 2 == 1, act=dt == torch.bfloat16 and D == 96, seed=D + V + H)
    close(scan(monkeypatch, True, rows, H, D, V, dt, **how), scan(monkeypatch, False, rows, H, D, V, dt, **how))


def run(qkv, tok, k_tok, state, rows, H, D, V, ones=False, act=False):
    from mini_inference_engine_b200.kernels import ops
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    T = sum(rows)
    dv = V + int(ones)
    state, out = state.clone(), torch.zeros(T, H * dv, device="cuda")
    ops.decay_scan(qkv, i32([0] * T), i32([sum(rows[:i]) for i in range(len(rows))]), i32(rows), i32([i + 1 for i in range(len(rows))]), state, out, num_heads=H, dim=D, vdim=V,
                   max_q_len=max(rows), tok_decay=tok, k_tok=k_tok, q_scale=0.125, q_lens=rows, ones=ones, act=act)
    torch.cuda.synchronize()
    return out.view(T, H, dv), state


def operands(rows, H, D, V, dt, least, seed=0, ones=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T = sum(rows)
    qkv = torch.randn(T, H * (2 * D + V), generator=g, device="cuda").to(dt)
    tok = least + (1 - least) * torch.rand(T, H, generator=g, device="cuda")
    return qkv, tok, torch.rand(T, H, generator=g, device="cuda"), torch.randn(len(rows) + 1, H, V + int(ones), D, generator=g, device="cuda")


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("least", [0.97, 0.5, 0.0])
def test_as_far_from_64_bits_as_token_by_token(monkeypatch, dt, least):
    from mini_inference_engine_b200.kernels import ops
    rows, H, D, V = [200, 130], 2, 128, 80
    qkv, tok, k_tok, state = operands(rows, H, D, V, dt, least)
    got = run(qkv, tok, k_tok, state, rows, H, D, V)
    monkeypatch.setattr(ops, "decay_chunks_take", lambda d: False)
    ref = run(qkv, tok, k_tok, state, rows, H, D, V)
    x = qkv.double()
    q, k, v = x[:, :H * D].view(-1, H, D) * 0.125, x[:, H * D:2 * H * D].view(-1, H, D) * k_tok.double()[:, :, None], x[:, 2 * H * D:].view(-1, H, V)
    out, end, at = torch.zeros_like(v), state.double().clone(), 0
    for r, n in enumerate(rows):
        S = end[r + 1].clone()
        for t in range(at, at + n):
            S = tok[t].double()[:, None, None] * S + v[t][:, :, None] * k[t][:, None, :]
            out[t] = (S * q[t][:, None, :]).sum(-1)
        end[r + 1] = S
        at += n
    for a, b, w in zip(got, ref, (out, end)):
        off = lambda t: ((t.double() - w).norm() / w.norm()).item()
        # measured over four seeds: outputs 0.93 to 1.13 times as far, states 0.90 to 1.13, with decays down to 0 (few terms a sum) 1.15 to 1.29
        assert off(a) <= 1.35 * off(b)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["value", "key", "query"])
def test_numbers_without_three_parts(monkeypatch, dt, what):
    """Beyond 2^127 and still finite: as the token-by-token kernel has them, token for token."""
    from mini_inference_engine_b200.kernels import ops
    rows, H, D, V = [150], 2, 32, 40
    qkv, tok, k_tok, state = operands(rows, H, D, V, dt, 0.9)
    qkv *= 1e-3
    col = dict(query=3, key=H * D + 3, value=2 * H * D + 3)[what]
    qkv[70, col] = 3e38
    got = run(qkv, tok, k_tok, state, rows, H, D, V)
    monkeypatch.setattr(ops, "decay_chunks_take", lambda d: False)
    ref = run(qkv, tok, k_tok, state, rows, H, D, V)
    for a, b in zip(got, ref):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.isfinite(a[:70]).all()
        ok = torch.isfinite(b)
        assert ((a - b).abs()[ok] <= 1.5e-5 * b[ok].abs().max()).all()
        quiet = ok & (b.abs() < 1e30)                          # what the large number does not reach keeps its digits
        assert ((a - b).abs()[quiet] <= 1.5e-5 * b[quiet].abs().max()).all()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what,bad", [("key", 3e38), ("key", float("inf")), ("key", float("nan")), ("value", 3e38)])
@pytest.mark.parametrize("H,V", [(12, 300), (2, 300), (9, 130), (1, 64)])
def test_column_of_ones_with_numbers_without_parts(monkeypatch, dt, what, bad, H, V):
    """Five tiles of value columns in three or five shares, three in three, one: the column of ones has one owner, whatever a share meets."""
    from mini_inference_engine_b200.kernels import ops
    rows, D = [150], 32
    qkv, tok, k_tok, state = operands(rows, H, D, V, dt, 0.9, ones=True)
    qkv *= 1e-3
    qkv[70, H * D + 3 if what == "key" else 2 * H * D + H * V - 1] = bad
    first = run(qkv, tok, k_tok, state, rows, H, D, V, ones=True)
    for _ in range(4):
        for a, b in zip(first, run(qkv, tok, k_tok, state, rows, H, D, V, ones=True)):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    monkeypatch.setattr(ops, "decay_chunks_take", lambda d: False)
    ref = run(qkv, tok, k_tok, state, rows, H, D, V, ones=True)
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(first[1]), kind(ref[1]))
    assert torch.isfinite(first[0][:70]).all()
    for a, b in zip(first, ref):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
        for some in (torch.isfinite(b) & (b.abs() < 1e30), torch.isfinite(b) & (b.abs() >= 1e30)):
            assert not some.any() or ((a - b).abs()[some] <= 1.5e-5 * b[some].abs().max()).all()


@pytest.mark.parametrize("dt,act", [(torch.float32, False), (torch.bfloat16, False), (torch.bfloat16, True)])
@pytest.mark.parametrize("what,bad", [("value", float("inf")), ("value", -float("inf")), ("value", float("nan")), ("value", 3.2e38), ("decay", float("inf")), ("decay", 3.4e38 / 2.0 ** 46)])
@pytest.mark.parametrize("D", [32, 128])
def test_infinite_values_and_decays_meet_no_parts(monkeypatch, dt, act, what, bad, D):
    """Keys of 1 have two parts of zero: a number that is not finite must not meet them.  States sign for sign as the token-by-token kernel has them; the keys in front of a
    large decay outgrow three parts only once it is multiplied in (3.4e38: finite, its nearest bfloat16 is not)."""
    from mini_inference_engine_b200.kernels import ops
    rows, H, V = [150], 2, 40
    qkv, tok, _, state = operands(rows, H, D, V, dt, 0.9)
    k_tok = torch.ones_like(tok)
    qkv[:, :H * D] *= 1e-3
    qkv[:, H * D:2 * H * D] = 1.0
    if what == "value":
        qkv[70, 2 * H * D + 3], tok[64:128] = bad, 1.0
    else:
        qkv[:, H * D:2 * H * D] = 2.0 ** 46
        qkv[:, 2 * H * D:] = qkv[:, 2 * H * D:].clamp(0.5, 1.0) * 1e-3
        state.abs_()
        tok[100], tok[101:128] = bad, 1.0
    how = dict(act=act)
    got = run(qkv, tok, k_tok, state, rows, H, D, V, **how)
    monkeypatch.setattr(ops, "decay_chunks_take", lambda d: False)
    ref = run(qkv, tok, k_tok, state, rows, H, D, V, **how)
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got[1]), kind(ref[1])), kind
    assert torch.equal(torch.isfinite(got[0]), torch.isfinite(ref[0]))
    for a, b in zip(got, ref):
        for some in (torch.isfinite(b) & (b.abs() < 1e30), torch.isfinite(b) & (b.abs() >= 1e30)):
            assert not some.any() or ((a - b).abs()[some] <= 1.5e-5 * b[some].abs().max()).all()
