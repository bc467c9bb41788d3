"""The channel delta rule's preparation four channels a lane, in runs of tokens, against the kernel that takes a token a block: rows that begin and end
inside a run, inputs older than the portion, head sizes with idle lanes, both types."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [[1], [1] * 9, [3, 1, 2, 8, 17, 5], [700, 900], [4000]])
@pytest.mark.parametrize("H,G,D,V", [(2, 2, 128, 128), (4, 2, 64, 32), (3, 1, 20, 12), (16, 16, 128, 128)])
@pytest.mark.parametrize("scale", [1.0, 1e20])                  # (1e20: sums of squares overflow, and unit vectors become zeros)
def test_runs_against_tokens(dt, rows, H, G, D, V, scale):
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(len(rows) + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, C = sum(rows), 2 * G * D + H * V
    if T > 1000 and H == 16:
        rows, T = [300, 260], 560
    proj, low = (rnd(T, -(-(C + H) // 8) * 8) * scale).to(dt), rnd(T, H * D + 4)
    taps, conv, a_log, bias = rnd(C, 4) * 0.5, rnd(len(rows) + 1, 3, C), rnd(H), rnd(H * D)
    lens = torch.tensor(rows, dtype=torch.int32, device="cuda")
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    token_row = torch.repeat_interleave(torch.arange(len(rows), dtype=torch.int32, device="cuda"), lens)
    slots = torch.tensor([len(rows) - i for i in range(len(rows))], dtype=torch.int32, device="cuda")
    results = []
    for shift in (0, 1):                                        # taps that do not start on 16 bytes: the kernel with a token a block
        t = torch.empty(C * 4 + 4, device="cuda")[shift:shift + C * 4].view(C, 4).copy_(taps)
        outs = [torch.zeros(T, n, device="cuda") for n in (G * D, G * D, H * V, H, H * D, G, H * D)]
        ops.delta_prepare(proj, low, t, conv, token_row, starts, slots, a_log, bias, *outs[:6], num_heads=H, num_kv_heads=G, dim=D, vdim=V, unit_eps=1e-6,
                          log_decay=outs[6])
        results.append(outs)
    torch.cuda.synchronize()
    for a, b in zip(*results):                                  # (sums of squares over a head in another order: a few units in the last place)
        assert torch.isfinite(a).all() and (a - b).abs().max() <= 2e-6 * b.abs().max()


@pytest.mark.parametrize("shift", [0, 1])
def test_a_decay_that_is_no_number_stays_none(shift):
    """Where the decay is NaN its logarithm is too (the chunks' kernels read that one), and nowhere else; decays of zero have a finite one."""
    from mini_inference_engine_b200.kernels import ops
    H, G, D, V, T = 2, 2, 64, 64, 70
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    C = 2 * G * D + H * V
    low = rnd(T, H * D + 4)
    low[16, 5], low[40], low[64, 70] = float("nan"), 1e30, float("nan")
    taps = torch.empty(C * 4 + 4, device="cuda")[shift:shift + C * 4].view(C, 4).copy_(rnd(C, 4))
    row, start, slot = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    outs = [torch.zeros(T, n, device="cuda") for n in (G * D, G * D, H * V, H, H * D, G, H * D)]
    ops.delta_prepare(rnd(T, C + 8), low, taps, rnd(2, 3, C), row, start, slot, rnd(H), rnd(H * D), *outs[:6], num_heads=H, num_kv_heads=G, dim=D, vdim=V,
                      unit_eps=1e-6, log_decay=outs[6])
    decay, log = outs[4], outs[6]
    assert decay.isnan().sum().item() == 2 and torch.equal(decay.isnan(), log.isnan())
    assert not decay[40].any() and (log[40] == -100.0).all()


def test_a_head_s_decay_that_is_no_number_stays_none():
    from mini_inference_engine_b200.kernels import ops
    H, G, D, V, T = 2, 1, 64, 64, 40
    g = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    C = 2 * G * D + H * V
    proj = rnd(T, C + H * V + 2 * H)
    a = proj[:, C + H * V:]
    a[16, 1], a[30, 0] = float("nan"), 1e30
    row, start, slot = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.ones(1, dtype=torch.int32, device="cuda")
    outs = [torch.zeros(T, n, device="cuda") for n in (G * D, G * D, H * V, H, H, H, G)]
    ops.delta_head_prepare(proj, rnd(4, C), rnd(2, 4, C), torch.arange(T, dtype=torch.int32, device="cuda"), row, start, slot, rnd(H), rnd(H), *outs,
                           num_heads=H, num_kv_heads=G, dim=D, vdim=V, unit_eps=1e-6)
    decay, log = outs[4], outs[5]
    assert decay.isnan().sum().item() == 1 and torch.equal(decay.isnan(), log.isnan())
    assert decay[30, 0] == 0 and log[30, 0] == -100.0
