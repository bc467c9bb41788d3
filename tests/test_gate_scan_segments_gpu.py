"""Exponential gates with a running maximum, a row cut into segments for the warps of a block, against 64 bits: row lengths at the edges of tiles and
segments, and the launch without segments; and the norm and gate that follow a linear-attention scan."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [[1, 32, 33], [5, 64, 31], [511, 512, 513], [2048], [40, 3000, 1]])
@pytest.mark.parametrize("cap", [0.0, 15.0])
def test_segments_against_64_bits(rows, cap):
    from mini_inference_engine_b200.kernels import ops
    H, T = 3, sum(rows)
    g = torch.Generator(device="cuda").manual_seed(T)
    z = torch.randn(T, 2 * H, generator=g, device="cuda") * 3
    bi, bf = torch.randn(H, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda") + 2
    lens = torch.tensor(rows, dtype=torch.int32, device="cuda")
    starts = torch.cumsum(lens, 0, dtype=torch.int32) - lens
    slots = torch.tensor([len(rows) - i for i in range(len(rows))], dtype=torch.int32, device="cuda")
    m0 = torch.rand(len(rows) + 1, H, generator=g, device="cuda") * 4
    zd = z.double()
    squash = (lambda t: cap * torch.tanh(t / cap)) if cap else (lambda t: t)
    gi, gf = squash(zd[:, :H] + bi.double()), torch.nn.functional.logsigmoid(squash(zd[:, H:] + bf.double()))
    want, m_end, at = [torch.zeros(T, H, dtype=torch.float64, device="cuda") for _ in range(3)], m0.double().clone(), 0
    for r, n in enumerate(rows):
        m = m_end[slots[r].item()]
        for t in range(at, at + n):
            new = torch.maximum(gf[t] + m, gi[t])
            want[0][t], want[1][t], want[2][t] = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new), new
            m = new
        m_end[slots[r].item()] = m
        at += n
    for longest in (None, max(rows), 1):                        # the last: one warp a row
        state = m0.clone()
        got = ops.gate_scan(z, bi, bf, cap, starts, lens, slots, state, H, longest)
        # a maximum is a sum of up to `rows` small terms carried in 32 bits: units in the last place of the largest, and the factors are its exponentials
        for a, w in zip(got, want):
            assert (a.double() - w).abs().max() <= 3e-5
        assert (state.double() - m_end).abs().max() <= 3e-5


@pytest.mark.parametrize("size,groups,w_len", [(256, 8, 2048), (100, 3, 100), (512, 1, 512), (513, 2, 1026), (64, 4, 64), (20, 5, 20)])
@pytest.mark.parametrize("normal", [False, True])
def test_norm_and_gate_of_groups_of_any_size(size, groups, w_len, normal):
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(size)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, stride = 37, size + int(normal)
    o, gate, w, m = rnd(T, groups * stride), rnd(T, groups * size + 3)[:, 2:2 + groups * size], rnd(w_len), rnd(T, groups).abs() if normal else None
    out = ops.group_norm_gate(o, gate, torch.zeros(T, groups * size, device="cuda"), groups=groups, size=size, eps=1e-5, weight=w, m=m)
    x = o.double().view(T, groups, stride)
    if normal:
        x = x[..., :size] / (torch.maximum(x[..., size].abs(), torch.exp(-m.double())) + 1e-6)[..., None]
    y = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).reshape(T, -1)
    y = y * w.double()[torch.arange(groups * size, device="cuda") % w_len] * torch.sigmoid(gate.double())
    assert (out.double() - y).abs().max() <= 4e-6 * y.abs().max()
