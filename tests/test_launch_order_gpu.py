"""Captured steps in which a kernel finds none of its rows, behind a slow product: the kernels behind it must not start before what is in front of it
has ended.  Against the same launches one at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def one_at_a_time(monkeypatch, step):
    """What ``step`` leaves when the device is idle in front of every launch."""
    from mini_inference_engine_b200.kernels import ops
    check = ops._check

    def then_wait(code, what):
        check(code, what)
        torch.cuda.synchronize()
    with monkeypatch.context() as m:
        m.setattr(ops, "_check", then_wait)
        out = [t.clone() for t in step()]
    torch.cuda.synchronize()
    return out


def replays(monkeypatch, x, inputs, clear, step):
    """``step`` captured and replayed over ``inputs`` in turn, each against its launches one at a time."""
    wanted = []
    for value in inputs:
        clear()
        x.copy_(value)
        wanted.append(one_at_a_time(monkeypatch, step))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for turn in range(12):
        clear()
        x.copy_(inputs[turn % len(inputs)])
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, wanted[turn % len(inputs)]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows", [[256], [250, 6], [130, 2]])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@torch.inference_mode()
def test_a_portion_with_no_short_row(monkeypatch, rows, dt):
    """The rows' lengths are unknown on the host, so the kernel for short rows runs and has none."""
    import numpy as np
    from test_getizen_parts_gpu import Harness, bind_random, build, rt_for
    from mini_inference_engine_b200.config import PartSpec
    from mini_inference_engine_b200.engine.batch import BatchRow
    rt, width = rt_for(dt), 4096
    mixer = build("mixer", "attention", hidden_size=width, num_heads=8, num_kv_heads=1, head_dim=64,
                  position=PartSpec("rope", dict(head_dim=64, rotary_dim=64, theta=1e4, max_position=512)))
    bind_random(mixer, rt, 1)
    h = Harness(mixer, rt)
    pages = iter(range(1, 64))
    ctx = h.builder.build([BatchRow([0] * n, 0, [np.array([next(pages) for _ in range(-(-n // h.builder.page_size))], dtype=np.int32)], 0, []) for n in rows])
    ctx.host["q_len"] = None
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.empty(sum(rows), width, dtype=dt, device=DEV)
    inputs = [torch.randn(sum(rows), width, generator=g, device=DEV).to(dt) for _ in range(3)]

    def clear():
        for t in h.storage.kv.values():
            t.zero_()
    replays(monkeypatch, x, inputs, clear, lambda: [mixer.forward(x, ctx, h.cache)] + list(h.storage.kv.values()))


@torch.inference_mode()
def test_a_recurrence_with_no_long_row(monkeypatch):
    """A launch laid out for long rows that holds none: the chunks' kernels have nothing to do, and what follows reads the short rows' outputs."""
    from mini_inference_engine_b200.kernels import ops
    from mini_inference_engine_b200.kernels.linear import linear
    H, D, V, rows = 4, 64, 64, [60, 64, 1, 33]
    T, width = sum(rows), 8192
    g = torch.Generator(device=DEV).manual_seed(5)
    w = torch.randn(H * (2 * D + 2 * V), width, generator=g, device=DEV) * width ** -0.5
    lens = torch.tensor(rows, dtype=torch.int32, device=DEV)
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    slots = torch.arange(1, len(rows) + 1, dtype=torch.int32, device=DEV)
    positions = torch.arange(T, dtype=torch.int32, device=DEV)
    decay, freq = torch.linspace(0.9, 0.99, H, device=DEV), torch.empty(0, device=DEV)
    state = torch.zeros(len(rows) + 1, H, V, D, device=DEV)
    x = torch.empty(T, width, device=DEV)
    inputs = [torch.randn(T, width, generator=g, device=DEV) for _ in range(3)]

    def step():
        qkvg = linear(x, w, None, torch.float32)
        o, gated = torch.empty(T, H * V, device=DEV), torch.empty(T, H * V, device=DEV)
        ops.retention_scan(qkvg, positions, starts, lens, slots, decay, freq, state, o, num_heads=H, dim=D, vdim=V, rot=0, k_scale=1.0, max_q_len=T, q_lens=None)
        ops.head_rms_gate(o, qkvg[:, H * (2 * D + V):], gated, H, V, 1e-5)
        return [gated, state]
    replays(monkeypatch, x, inputs, lambda: state.zero_(), step)
