"""The float32 product on the tensor cores (operands split into three bfloat16 parts) against 64 bits, at the edges of its tiles and
slabs, and where a number is not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(M, N, K, seed=0, spread=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    if spread:                                                             # magnitudes over 2^-20 .. 2^20
        x, w = (t * torch.exp2(torch.randint(-20, 21, t.shape, generator=g, device="cuda").float()) for t in (x, w))
    return x, w, torch.randn(N, generator=g, device="cuda")


def check(got, x, w, bias):
    """A float32 dot product of K terms in any order, rounded at every addition, is within K u sum |x||w| of the true one, and within
    about sqrt(K) u of it for most: 4 sqrt(K) u sum |x||w| with u = 2^-24."""
    want = x.double() @ w.double().t()
    room = 4 * x.shape[1] ** 0.5 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    if bias is not None:
        want, room = want + bias.double(), room + 2.0 ** -23 * (want.abs() + bias.double().abs())
    assert ((got.double() - want).abs() <= room).all()


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("M,N,K", [(9, 128, 128), (17, 2048, 2048), (63, 256, 64 * 9), (64, 257, 130), (65, 255, 1000), (128, 1000, 129),
                                   (129, 512, 4099), (255, 264, 257), (256, 768, 320), (257, 2048, 512), (600, 130, 2050)])
def test_any_sizes(M, N, K, spread):
    from mini_inference_engine_b200.kernels import gemm_split, gemm_tc
    x, w, bias = operands(M, N, K, M + N, spread)
    for b in (None, bias, bias.to(torch.bfloat16)):
        got = gemm_split.gemm_split(x, w, torch.empty(M, N, device="cuda"), b)
        torch.cuda.synchronize()
        gemm_tc.check_error()
        check(got, x, w, b)


@pytest.mark.parametrize("K", [128, 512, 2048])
@pytest.mark.parametrize("kind", ["equal", "just above", "just below", "one sign", "both signs"])
def test_no_further_from_64_bits_than_float32_sums(kind, K):
    """Significands whose parts are as large as they get, products of one sign, whose errors add up, and ordinary numbers: the 2-norm of the error is no larger
    than that of chains of fused multiply-adds, or than half a unit in the last place of the results, which both sides lose at the end."""
    from mini_inference_engine_b200.kernels import gemm_split, ops
    M, N = 200, 320
    g = torch.Generator(device="cuda").manual_seed(K)
    few = lambda *s: torch.randint(0, 8, s, generator=g, device="cuda").float() * 2.0 ** -23
    make = {"equal": lambda *s: torch.full(s, 1.0 + 2.0 ** -7 - 2.0 ** -23, device="cuda"), "just above": lambda *s: 1.0 + 2.0 ** -8 - few(*s),
            "just below": lambda *s: 1.0 - 2.0 ** -9 - few(*s) / 2, "one sign": lambda *s: 1.0 + torch.rand(*s, generator=g, device="cuda"),
            "both signs": lambda *s: torch.randn(*s, generator=g, device="cuda")}[kind]
    x, w = make(M, K), make(N, K)
    want = x.double() @ w.double().t()
    off = lambda t: ((t.double() - want).norm() / want.norm()).item()
    split, chain = off(gemm_split.gemm_split(x, w, torch.empty(M, N, device="cuda"))), off(ops.gemm_simt(x, w, torch.empty(M, N, device="cuda")))
    print(f"{kind}, K {K}: split {split:.3g}, fused multiply-adds {chain:.3g}")
    assert split <= max(chain, 2.0 ** -24)


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("splits", [1, 3, 8])
def test_every_tile_and_share_of_k(bn, splits):
    from mini_inference_engine_b200.kernels import gemm_split
    x, w, bias = operands(300, 700, 64 * 11 + 5, bn)
    check(gemm_split.gemm_split(x, w, torch.empty(300, 700, device="cuda"), bias, force=(bn, splits)), x, w, bias)


def test_operands_in_slabs(monkeypatch):
    from mini_inference_engine_b200.kernels import gemm_split
    monkeypatch.setattr(gemm_split, "W_SLAB_BYTES", 1)
    monkeypatch.setattr(gemm_split, "X_SLAB_BYTES", 1)
    x, w, bias = operands(520, 600, 200)
    check(gemm_split.gemm_split(x, w, torch.empty(520, 600, device="cuda"), bias), x, w, bias)


def test_operands_that_start_anywhere():
    from mini_inference_engine_b200.kernels import gemm_split
    x, w, _ = operands(40, 256, 200)
    xo, wo = torch.empty(40 * 200 + 1, device="cuda")[1:].view(40, 200).copy_(x), torch.empty(256 * 200 + 3, device="cuda")[3:].view(256, 200).copy_(w)
    out = torch.empty(40 * 256 + 1, device="cuda")[1:].view(40, 256)
    check(gemm_split.gemm_split(xo, wo, out), x, w, None)


@pytest.mark.parametrize("force", [(64, 1), (128, 2)])
def test_numbers_that_are_not_finite_or_overflow(force):
    """Infinities, NaN and sums beyond the largest float32 come out as the CUDA-core product leaves them."""
    from mini_inference_engine_b200.kernels import gemm_split, ops
    x, w, _ = operands(70, 300, 512)
    x[3, 5], x[7, 9], w[11, 100], x[50], w[20, 0], x[60, 0] = float("inf"), float("nan"), -float("inf"), 3e38, 0.0, float("inf")
    got = gemm_split.gemm_split(x, w, torch.empty(70, 300, device="cuda"), force=force)
    want = ops.gemm_simt(x, w, torch.empty(70, 300, device="cuda"))
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(want))
    fine = torch.isfinite(want)
    fine[50] = False                                                       # (finite sums of huge terms: nothing to compare but that they are finite)
    assert ((got - want).abs()[fine] <= 1e-4 * 512 ** 0.5).all()


@pytest.mark.parametrize("what", ["nan", "inf", "overflow", "a column"])
@pytest.mark.parametrize("force", [(64, 1), (256, 1), (128, 3)])
def test_many_outputs_that_are_not_finite(what, force):
    """A step of such numbers is what the CUDA-core product leaves, and takes no more than a few times that product's time (seen: 4 to 7 times, the latter with
    tiles that only a third of the SMs have; with an output after the other in a thread the limit below is passed in every case)."""
    from mini_inference_engine_b200.kernels import gemm_split, gemm_tc, ops
    M, N, K = 640, 2048, 1024
    x, w, bias = operands(M, N, K, 3)
    if what == "nan":
        x.fill_(float("nan"))
    elif what == "inf":
        x[:] = float("inf")
    elif what == "overflow":
        x, w = x.abs() * 1e20 + 1e20, w.abs() * 1e19 + 1e19
    else:
        w[:, 17] = -float("inf")
    got, want = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    split, plain = lambda: gemm_split.gemm_split(x, w, got, bias, force=force), lambda: ops.gemm_simt(x, w, want, bias)
    times = []
    for fn in (split, plain):
        fn()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(3):
            fn()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) / 3)
    gemm_tc.check_error()
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(got), kind(want))
    assert not torch.isfinite(want).any()
    print(f"{what}, {force}: {times[0]:.3f} ms, the CUDA-core product {times[1]:.3f} ms")
    assert times[0] <= 16 * times[1]


@pytest.mark.parametrize("down,up", [(-104, 90), (-113, 100), (-120, 110), (-128, 115), (-140, 120)])
def test_numbers_below_the_range_of_their_parts(down, up):
    """Operands down to float32's last bit, times large ones: nothing of them is lost."""
    from mini_inference_engine_b200.kernels import gemm_split
    x, w, _ = operands(70, 300, 512, 7)
    x[5] = 0.0
    x[9, ::2] = 0.0
    x, w = x * 2.0 ** down, w * 2.0 ** up
    check(gemm_split.gemm_split(x, w, torch.empty(70, 300, device="cuda")), x, w, None)
    check(gemm_split.gemm_split(w, x, torch.empty(300, 70, device="cuda"), force=(64, 2)), w, x, None)


def test_the_runtime_takes_it_for_prompts_in_float32():
    from mini_inference_engine_b200.kernels import gemm_split
    from mini_inference_engine_b200.kernels.linear import linear
    assert gemm_split.takes(200, 256, 256) and not gemm_split.takes(8, 2048, 2048) and not gemm_split.takes(200, 64, 64)
    x, w, bias = operands(200, 256, 256)
    got = linear(x, w, bias, torch.float32)
    assert torch.equal(got, gemm_split.gemm_split(x, w, torch.empty_like(got), bias))
    check(got, x, w, bias)


def test_its_first_use_may_fall_into_a_capture():
    """A process whose first product of this kind is captured (a portion that ran on the CUDA cores is captured at its padded length)."""
    import os
    import subprocess
    import sys
    code = """
import torch
from mini_inference_engine_b200.kernels import gemm_split, gemm_tc
x, w, out = torch.randn(32, 256, device="cuda"), torch.randn(512, 256, device="cuda"), torch.empty(32, 512, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    gemm_split.gemm_split(x, w, out)
graph.replay()
torch.cuda.synchronize()
gemm_tc.check_error()
want = x.double() @ w.double().t()
assert ((out.double() - want).norm() / want.norm()).item() < 1e-6
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
