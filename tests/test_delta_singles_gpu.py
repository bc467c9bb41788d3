"""The gated delta rule's rows of one new token without the scan's ring, against the scan: columns that end inside a block, key heads shared by heads,
rows that belong to another kernel and rows without a token, key sizes that only the scan takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [48, 64, 96, 128, 160])
@pytest.mark.parametrize("Dv", [1, 32, 40, 128])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("lens", [[1], [1] * 33, [1, 130, 1, 0, 200, 1]])
def test_single_tokens_like_the_scan(D, Dv, per_channel, lens):
    from mini_inference_engine_b200.kernels import ops
    H, G, below = 6, 2, 112
    T, rows = sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(D + Dv + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    qn, kn = (torch.nn.functional.normalize(rnd(T, G, D), dim=-1).reshape(T, G * D) for _ in "qk")
    vn, beta = rnd(T, H * Dv), rnd(T, H).sigmoid()
    decay = rnd(T, H * D if per_channel else H).sigmoid()
    kq = (qn.view(T, G, D) * kn.view(T, G, D)).sum(-1)
    start = torch.tensor([sum(lens[:i]) for i in range(rows)], dtype=torch.int32, device=DEV)
    count = torch.tensor(lens, dtype=torch.int32, device=DEV)
    slots = torch.randperm(rows + 3, generator=torch.Generator().manual_seed(1))[:rows].int().to(DEV)
    first = rnd(rows + 3, H, Dv, D)
    got = []
    for singles in (False, True):
        state, out = first.clone(), torch.full((T, H * Dv), 7.0, device=DEV)
        ops.delta_scan(qn, kn, vn, beta, decay, kq, start, count, slots, state, out, num_heads=H, num_kv_heads=G, dim=D, vdim=Dv, below=below, singles=singles)
        got.append((state, out))
    # the same operations but for one: the decayed S^T k is rounded before it is taken off v, or the subtraction is one fused operation.  That is 2^-24 of
    # |S^T k| <= sqrt(D) max |S| in u; k, q and beta are at most 1, and the sums that take u round once more each
    near = lambda a, b: ((a - b).abs() <= 2.0 ** -22 * (1 + vn.abs().max() + D ** 0.5 * first.abs().max())).all()
    assert near(got[0][0], got[1][0]) and near(got[0][1], got[1][1])
    other = [i for i, n in enumerate(lens) if n != 1]          # rows that are not the kernel's stay as they are, to the bit
    untouched = sorted(set(range(rows + 3)) - {int(slots[i]) for i in range(rows) if lens[i] == 1})
    assert torch.equal(got[1][0][untouched], first[untouched])
    for i in other:
        assert (got[1][1][int(start[i]):int(start[i]) + lens[i]] == 7.0).all()
    # and the recurrence itself in 64 bits, for the first row
    s, k, q = first[slots[0].long()].double(), kn[0].view(G, D).double().repeat_interleave(H // G, 0), qn[0].view(G, D).double().repeat_interleave(H // G, 0)
    s = s * decay[0].double().view(H, 1, -1)
    u = beta[0].double()[:, None] * (vn[0].view(H, Dv).double() - (s * k[:, None]).sum(-1))
    s = s + u[..., None] * k[:, None]
    assert ((got[1][0][slots[0].long()].double() - s).abs() <= 2.0 ** -22 * (1 + D / 16) * (1 + s.abs().max())).all()
    o = (s * q[:, None]).sum(-1).view(-1)
    assert ((got[1][1][0].double() - o).abs() <= 2.0 ** -22 * (1 + D / 16) * (1 + s.abs().max() * D ** 0.5)).all()
