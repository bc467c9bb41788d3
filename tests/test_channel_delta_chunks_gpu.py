"""The gated delta rule with a decay per key channel in chunks of 64 tokens against 64 bits and against the token-by-token kernel: row lengths at
the edges of chunks, key and value sizes, heads that share keys, decays from none to all at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(rows, H, G, D, V, decays, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T = sum(rows)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)
    q, k = unit(rnd(T, G, D)) * D ** -0.5, unit(rnd(T, G, D))
    if decays == "mild":
        log = -torch.rand(T, H, D, generator=g, device="cuda") * 0.1
    elif decays == "mixed":                                   # from none to a factor of e^-40 a token, channel by channel
        log = -torch.exp(rnd(T, H, D) * 2.5 - 2.0).clamp(max=40.0)
        log[rnd(T, H, D) > 1.2] = 0.0
    else:                                                     # all gone at some tokens
        log = -torch.rand(T, H, D, generator=g, device="cuda") * 0.5
        log[3::19] = -100.0
    beta = torch.sigmoid(rnd(T, H))
    lens = torch.tensor(rows, dtype=torch.int32, device="cuda")
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    slots = torch.tensor([len(rows) - i for i in range(len(rows))], dtype=torch.int32, device="cuda")
    state = rnd(len(rows) + 1, H, V, D) * 0.5
    return q, k, rnd(T, H, V), beta, log, starts, lens, slots, state


def exact(rows, q, k, v, beta, log, slots, state, H, G):
    q, k, v, beta, g, S_all = (t.double() for t in (q, k, v, beta, torch.exp(log), state.clone()))
    o, at = torch.zeros_like(v), 0
    rep = lambda t: t.repeat_interleave(H // G, 0)
    for r, n in enumerate(rows):
        S = S_all[slots[r].item()]
        for t in range(at, at + n):
            S = S * g[t][:, None, :]
            u = beta[t][:, None] * (v[t] - (S * rep(k[t])[:, None, :]).sum(-1))
            S = S + u[:, :, None] * rep(k[t])[:, None, :]
            o[t] = (S * rep(q[t])[:, None, :]).sum(-1)
        S_all[slots[r].item()] = S
        at += n
    return o, S_all


def run(rows, q, k, v, beta, log, starts, lens, slots, state, H, G, D, V, min_len=1, known=True, token_by_token=False, a_head=False):
    from mini_inference_engine_b200.kernels import ops
    T = sum(rows)
    state, out = state.clone(), torch.zeros(T, H * V, device="cuda")
    flat = lambda t: t.reshape(T, -1).contiguous()
    sizes = dict(num_heads=H, num_kv_heads=G, dim=D, vdim=V)
    decay = torch.exp(log)
    if a_head:                                                # one decay per head: the first channel's
        ops.delta_chunks(flat(q), flat(k), flat(v), beta, log[:, :, 0].contiguous(), starts, lens, slots, state, out, min_len=min_len, **sizes)
    elif token_by_token:
        kq = flat((q * k).sum(-1))
        ops.delta_scan(flat(q), flat(k), flat(v), beta, flat(decay), kq, starts, lens, slots, state, out, **sizes)
    else:
        long = [n for n in rows if n >= min_len]
        ops.delta_chunks(flat(q), flat(k), flat(v), beta, flat(log), starts, lens, slots, state, out, min_len=min_len,
                         work=(len(long), sum(long)) if known else None, decay=flat(decay), **sizes)
    torch.cuda.synchronize()
    return out.view(T, H, V), state


@pytest.mark.parametrize("decays", ["mild", "mixed", "gone"])
@pytest.mark.parametrize("H,G,D,V,rows", [(2, 2, 128, 128, [64, 65, 130]), (4, 2, 64, 48, [1, 16, 17, 63, 200]), (2, 1, 100, 20, [90, 33]), (1, 1, 4, 3, [70]),
                                          (3, 3, 68, 16, [128, 127])])
def test_chunks_against_64_bits(decays, H, G, D, V, rows):
    """No further from 64 bits than twice the token-by-token kernel or a few float32 roundings of the largest value."""
    args = operands(rows, H, G, D, V, decays, H + D + V)
    q, k, v, beta, log, starts, lens, slots, state = args
    want = exact(rows, q, k, v, beta, log, slots, state, H, G)
    got, ref = run(rows, *args, H, G, D, V), run(rows, *args, H, G, D, V, token_by_token=True)
    for a, b, w in zip(got, ref, want):
        off = lambda t: (t.double() - w).abs().max().item()
        assert torch.isfinite(a).all() and off(a) <= max(2.0 * off(b), 32 * 2.0 ** -24 * w.abs().max().item())


@pytest.mark.parametrize("known", [True, False])
def test_short_rows_are_left_alone(known):
    rows, H, G, D, V = [5, 150, 1, 64], 2, 2, 32, 24
    args = operands(rows, H, G, D, V, "mild")
    out, state = run(rows, *args, H, G, D, V, min_len=64, known=known)
    ref, ref_state = run(rows, *args, H, G, D, V, token_by_token=True)
    assert not out[:5].any() and not out[155].any()
    for r, slot in enumerate(args[7].tolist()):
        if rows[r] < 64:
            assert torch.equal(state[slot], args[8][slot])
        else:
            assert (state[slot] - ref_state[slot]).abs().max() <= 1e-5 * ref_state.abs().max()
    for lo, hi in ((5, 155), (156, 220)):
        assert (out[lo:hi] - ref[lo:hi]).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("a_head", [False, True])
@pytest.mark.parametrize("at", [0, 15, 64, 75, 85, 103, 112, 127, 139])
@pytest.mark.parametrize("what", ["key", "value"])
def test_a_token_that_is_not_finite_spoils_only_what_follows(what, at, a_head):
    rows, H, G, D, V = [140, 80], 2, 2, 32, 24
    args = operands(rows, H, G, D, V, "mild")
    args[1 if what == "key" else 2][at] = float("nan")
    out, _ = run(rows, *args, H, G, D, V, a_head=a_head)
    assert torch.isfinite(out[:at]).all() and torch.isfinite(out[140:]).all() and not torch.isfinite(out[at:140]).any()


@pytest.mark.parametrize("a_head", [False, True])
@pytest.mark.parametrize("H,G", [(5, 5), (6, 3), (4, 1)])
def test_some_heads_at_a_time(monkeypatch, H, G, a_head):
    """Scratch memory for one key head's heads, or two, at a time: every number as with all at once."""
    from mini_inference_engine_b200.kernels import ops
    rows, D, V = [100, 65, 3], 32, 24
    args = operands(rows, H, G, D, V, "mixed")
    whole = run(rows, *args, H, G, D, V, a_head=a_head)
    sizes, empty = [], torch.empty
    for key_heads in (1, 2):
        with monkeypatch.context() as m:
            m.setattr(ops, "_heads_a_pass", lambda heads, bytes_a_head: min(heads, key_heads))
            m.setattr(ops.torch, "empty", lambda *s, **k: (sizes.append(s[0]), empty(*s, **k))[1])
            got = run(rows, *args, H, G, D, V, a_head=a_head)
        assert all(torch.equal(a, b) for a, b in zip(got, whole))
    assert sizes[0] * G == sizes[1] * G // min(2, G)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_the_mixer_in_portions_of_any_length(dt):
    """Whole, in long and short portions, and beside decoding rows: the same outputs."""
    from test_getizen_parts_gpu import Harness, bind_random, build, inputs, rt_for, run_in_portions
    rt = rt_for(dt)
    mixer = build("mixer", "channel_delta", hidden_size=64, num_heads=2, num_kv_heads=2, dim=32, vdim=32, taps=4, eps=1e-5)
    bind_random(mixer, rt, 3)
    x = inputs(300, 64, 1, dt)
    whole = run_in_portions(Harness(mixer, rt), x, [300])
    tokens = run_in_portions(Harness(mixer, rt), x, [50] * 6)
    mixed = run_in_portions(Harness(mixer, rt), x, [1, 130, 2, 112, 55])
    bound = (2e-5 if dt == torch.float32 else 2e-2) * whole.abs().max()
    assert (whole - tokens).abs().max() <= bound and (whole - mixed).abs().max() <= bound
