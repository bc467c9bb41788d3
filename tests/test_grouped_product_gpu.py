"""The product of row ranges with a matrix each: groups of no row, one row and around a tile's 256, rows behind the last group, sums and columns that end inside a
tile, matrices stacked and side by side, a group whose weights are not numbers beside others, more tiles than pairs of SMs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"

SIZES = {"one": [5], "edges": [0, 1, 255, 0, 256, 257, 3, 0], "many": [33] * 40, "tall": [1500, 0, 700], "none": [0, 0]}


@pytest.mark.parametrize("sizes", list(SIZES))
@pytest.mark.parametrize("K,N", [(8, 8), (64, 256), (72, 264), (960, 2048), (1000, 520)])
@pytest.mark.parametrize("side_by_side", [False, True])
@pytest.mark.parametrize("relu2", [False, True])
def test_grouped_product(sizes, K, N, side_by_side, relu2):
    from mini_inference_engine_b200.kernels import ops
    counts = SIZES[sizes]
    E, behind = len(counts), 7
    R = sum(counts) + behind
    g = torch.Generator(device=DEV).manual_seed(K + N + E)
    x = torch.randn(R, K, generator=g, device=DEV).bfloat16()
    w = torch.randn(E, N, K, generator=g, device=DEV).bfloat16()
    lost = E // 2 if E > 1 else None
    if lost is not None:
        w[lost] = float("nan")                                 # stays in its own group's rows
    if side_by_side:                                           # [N, E K]: group e's matrix is the columns from e K
        flat = w.permute(1, 0, 2).reshape(N, E * K).contiguous()
        b = torch.as_strided(flat, (E, K, N), (K, 1, E * K))
    else:
        b = w.transpose(1, 2)
    ends = torch.tensor(counts).cumsum(0).int().to(DEV)
    weight = torch.rand(R, generator=g, device=DEV) + 0.5 if relu2 else None
    assert ops.grouped_fits(x, b, ends)
    out = ops.grouped_linear(x, b, ends, relu2_weight=weight)
    assert out.shape == (R, N) and out.dtype == torch.bfloat16
    at = 0
    for e, n in enumerate(counts):
        rows, at = slice(at, at + n), at + n
        if e == lost or n == 0:
            continue
        a, m = x[rows].double(), w[e].double()
        want, scale = a @ m.t(), a.abs() @ m.abs().t()
        error = 2.0 ** -21 * scale                             # the float32 sum: the tensor cores' partial sums keep 22 bits and more of their largest term
        if relu2:
            f = weight[rows].double()[:, None]
            error = f * (2 * want.abs() * error + error * error)
            want = f * want.clamp_min(0) ** 2
        assert ((out[rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + error + 1e-30).all(), e


def test_operands_that_the_kernel_refuses_go_to_the_library():
    from mini_inference_engine_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(64, 64, generator=g, device=DEV).bfloat16()
    w = torch.randn(2, 64, 32, generator=g, device=DEV).bfloat16()              # N innermost
    ends = torch.tensor([40, 64], dtype=torch.int32, device=DEV)
    assert not ops.grouped_fits(x, w, ends)
    out = ops.grouped_linear(x, w, ends)
    want = torch.cat([x[:40].double() @ w[0].double(), x[40:].double() @ w[1].double()])
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
