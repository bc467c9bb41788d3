"""The linear-attention step of single tokens in one launch against the scan's kernels: rotation, activation, decays per head and per token, the column of ones, norm
and gate, key sizes with idle lanes, value sizes off the tile, both types, and which steps the mixers hand it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V,rot", [(2, 128, 256, 128), (3, 64, 40, 16), (1, 20, 9, 8), (8, 100, 130, 0), (2, 4, 300, 0)])
@pytest.mark.parametrize("rows", [1, 5, 33])
@pytest.mark.parametrize("what", ["plain", "norm", "act", "tokens"])
def test_step_against_scan(dt, H, D, V, rot, rows, what):
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(H + D + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ones, act = what == "tokens", what == "act"
    rot = 0 if act else rot
    dv = V + int(ones)
    qkv = rnd(rows, -(-H * (2 * D + 2 * V) // 8) * 8).to(dt)
    state = rnd(rows + 1, H, dv, D)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts, lens, slots, pos = i32(list(range(rows))), i32([1] * rows), i32([rows - i for i in range(rows)]), i32([7 * i + 3 for i in range(rows)])
    how = dict(num_heads=H, dim=D, vdim=V, act=act, ones=ones, k_scale=D ** -0.5, q_scale=0.7 if ones else 1.0,
               freq=torch.rand(rot // 2, generator=g, device="cuda") if rot else None, rot=rot)
    if ones:
        how.update(tok_decay=torch.rand(rows, H, generator=g, device="cuda"), k_tok=torch.rand(rows, H, generator=g, device="cuda"))
    else:
        how.update(decay=torch.rand(H, generator=g, device="cuda"))
    want_state, o = state.clone(), torch.zeros(rows, H * dv, device="cuda")
    ops.decay_scan(qkv, pos, starts, lens, slots, want_state, o, max_q_len=1, **how)
    if what == "norm":
        gate = qkv[:, H * (2 * D + V):H * (2 * D + 2 * V)]
        want = ops.head_rms_gate(o, gate, torch.zeros(rows, H * V, dtype=dt, device="cuda"), H, V, 1e-5)
        got = ops.decay_step(qkv, pos, starts, slots, state, gate=gate, gated=torch.zeros_like(want), eps=1e-5, **how)
    else:
        want = o
        got = ops.decay_step(qkv, pos, starts, slots, state, torch.zeros_like(o), **how)
    # the state entry by entry the same operations (the compiler's own sin and cos aside); a read-out of D terms in another order
    assert (state - want_state).abs().max() <= 1e-6 * want_state.abs().max()
    tol = 2e-5 if got.dtype == torch.float32 else 8e-3
    assert torch.isfinite(got.float()).all() and (got.float() - want.float()).abs().max() <= tol * want.float().abs().max()


@pytest.mark.parametrize("kind", ["retention", "lightning_attention", "matrix_memory"])
def test_the_mixers_take_it_for_steps_of_single_tokens(kind, monkeypatch):
    from test_getizen_parts_gpu import Harness, bind_random, build, inputs, rt_for
    from mini_inference_engine_b200.kernels import ops
    rt = rt_for(torch.float32)
    more = dict(retention=dict(decay=[0.9, 0.7], rot_dims=16, rot_base=1e4), lightning_attention=dict(decay=[0.9, 0.7]), matrix_memory=dict(gate_cap=15.0))[kind]
    mixer = build("mixer", kind, hidden_size=48, num_heads=2, dim=32, vdim=40, eps=1e-5, **more)
    bind_random(mixer, rt, 3)
    x = inputs(12, 48, 1, torch.float32)
    calls = []
    step = ops.decay_step
    monkeypatch.setattr(ops, "decay_step", lambda *a, **k: calls.append(1) or step(*a, **k))
    results = []
    for single in (True, False):
        h = Harness(mixer, rt)
        a, b = h.new(), h.new()
        h.step([(a, x[:5]), (b, x[5:7])])
        if not single:
            monkeypatch.setattr(ops, "decay_step_takes", lambda *a: False)
        results.append(torch.cat(h.step([(a, x[7:8]), (b, x[8:9])]) + h.step([(b, x[9:10]), (a, x[10:11])])))
    assert len(calls) == 2
    assert (results[0] - results[1]).abs().max() <= 2e-5 * results[1].abs().max()
