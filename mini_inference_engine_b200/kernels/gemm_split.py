"""The float32 product on the tensor cores (``csrc/gemm_split_tc.cu``): which sizes it takes, its plan and its launches.

Both operands are split into three bfloat16 planes in scratch memory, in slabs, so that the scratch is bounded whatever the weight's size."""
from __future__ import annotations

import ctypes

import torch

from . import build, ops
from .device import num_sms

# Device time against the CUDA-core product, B200, weights from memory (L2 overwritten in front of every product), us, CUDA cores : here, at 9 / 16 / 17 / 32 tokens.
# Up to 16 tokens its row-streaming kernel runs, which reads w once per eight tokens and is the faster one where w has rows for all SMs many times over, or is small:
#   1,024 x 128 (outputs x K) 4 : 11 / 4 : 11 / 14 : 11 / 14 : 11    1,024 x 1,024 19 : 15 / 19 : 16 / 102 : 15 / 103 : 16 (w in L2: 9 : 14 up to 16 tokens)
#   2,048 x 2,048 36 : 23 / 36 : 24 / 209 : 24 / 214 : 24            4,096 x 2,048 45 : 35 / 52 : 36 / 208 : 36 / 217 : 36
#   11,264 x 2,048 89 : 88 / 115 : 88 / 235 : 88 / 239 : 88          2,048 x 5,632 90 : 46 / 91 : 46 / 583 : 46 / 605 : 47
#   5,632 x 4,096 119 : 87 / 165 : 88 / 428 : 87 / 433 : 88          32,000 x 2,048 207 : 251 / 228 : 251 / 327 : 251 / 334 : 252
# (taken with the parts' first form; the present one takes 12 to 14 less for 11,264 x 2,048.)  From 17 tokens on every size from 128 x 128 on: 13 : 11.  More tokens: 509 x 11,264 x 2,048
# 1,008 : 140 - 143, 509 x 2,048 x 5,632 1,195 : 78, 2,048 x 11,264 x 2,048 2,707 : 403; smaller ones: 2,000 x 128 x 128 40 : 16, 2,000 x 64 x 64 12 : 15 (three launches instead of one).
MIN_TOKENS = 9
MIN_K = 128
MIN_WEIGHT = 1 << 14
FEW_TOKENS = 16                       # up to this many tokens ...
FEW_MIN_WEIGHT = 1 << 22              # ... from this size on (smaller ones are likely to be in L2) ...
FEW_MAX_ASPECT = 6                    # ... and up to this many outputs per entry of K
W_SLAB_BYTES = 144 << 20              # planes of the weight rows that are in scratch at a time (a slab of 23 M numbers: one
                                      # gate|up matrix of 2 x 5,632 x 2,048 in one go)
X_SLAB_BYTES = 48 << 20
PARTIAL_BYTES = 48 << 20


def takes(M: int, N: int, K: int) -> bool:
    if M <= FEW_TOKENS and (N * K < FEW_MIN_WEIGHT or N > FEW_MAX_ASPECT * K):
        return False
    return M >= MIN_TOKENS and K >= MIN_K and N * K >= MIN_WEIGHT


def plan(M: int, N: int, K: int, only: int = 0) -> tuple:
    """(tokens a tile, shares of K, tiles of 256 rows of w in front that take all of K at once): the plan with the least estimated time, in cycles
    (``only``: of those with this many tokens a tile).
    Measured: a 64-wide chunk of K takes a pair of SMs 1,900, 2,250 or 3,850 cycles with 64, 128 or 256 tokens (the 24 MMAs alone 770, 1,540, 3,070:
    with 256 tokens only two accumulators fit tensor memory, and the way from a full one to an empty one is as long as the MMAs); an item's start and
    end 3,000; shares of K write and read M x (rows they cover) partial sums each at some 2,500 bytes a cycle, in a launch more.  The tiles in front
    fill whole waves of pairs; those behind them would leave most pairs idle, so it is they that are worth shares (all tiles whole : with shares behind, us,
    B200, tokens x outputs x K: 509 x 11,264 x 2,048 161 : 140 - 143; 1,000 x 5,632 x 2,048 146 : 127; 1,000 x 2,560 x 2,048 73 : 66; 700 x 32,000 x 2,048 545 : 501)."""
    pairs = max(1, num_sms() // 2)
    chunks, tiles_n = -(-K // 64), -(-N // 256)
    best = None
    for bn, cycles in ((256, 3850), (128, 2250), (64, 1900)):
        if only and bn != only:
            continue
        tiles_m = -(-M // bn)
        for whole in {0, tiles_m * tiles_n // pairs * pairs // tiles_m}:
            rest = tiles_n - whole
            front = -(-whole * tiles_m // pairs) * (chunks * cycles + 3000)
            for splits in (1, 2, 3, 4, 5, 6, 8):
                sums = splits * M * min(rest * 256, N) * 4
                if (whole and (splits > 1) != (rest > 0)) or splits > max(1, chunks // 4) or (splits > 1 and sums > PARTIAL_BYTES):
                    continue
                per = -(-chunks // splits)
                t = front + -(-tiles_m * rest * splits // pairs) * (per * cycles + 3000) + (sums * 2 / 2500 + 4000 if splits > 1 else 0)
                if best is None or t < best[0]:
                    best = (t, bn, splits, whole if splits > 1 else 0)
    return best[1:]


def _split(lib, t: torch.Tensor, block: int) -> torch.Tensor:
    """The planes of ``t`` in blocks of ``block`` rows, an even number of them (a pair of SMs takes two)."""
    rows, K = t.shape
    blocks = -(-rows // (2 * block)) * 2
    planes = torch.empty(-(-K // 64) * blocks * 3 * block * 64, dtype=torch.bfloat16, device=t.device)
    ops._check(lib.mie_split3(ops._ptr(t), ops._ptr(planes), rows, K, block, blocks, ops._stream()), "split3")
    return planes


def gemm_split(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, bias: torch.Tensor | None = None, force: tuple | None = None) -> torch.Tensor:
    """out[M, N] = x[M, K] @ w[N, K]^T (+ bias), all float32 and contiguous, at the precision of float32 products."""
    (M, K), N = x.shape, w.shape[0]
    ops._need(x.dtype == w.dtype == out.dtype == torch.float32, "the split product takes float32 operands and leaves float32")
    ops._need(w.shape[1] == K and tuple(out.shape) == (M, N), f"gemm shapes: x {tuple(x.shape)}, w {tuple(w.shape)}, out {tuple(out.shape)}")
    ops._need(x.is_contiguous() and w.is_contiguous() and out.is_contiguous(), "gemm operands must be contiguous")
    lib = ops.load("gemm_split_tc")
    Kp = -(-K // 64) * 64
    w_rows = max(256, W_SLAB_BYTES // (6 * Kp) // 256 * 256)
    x_rows = max(256, X_SLAB_BYTES // (6 * Kp) // 256 * 256)
    first = (*force, 0)[:3] if force else plan(min(M, x_rows), min(N, w_rows), K)
    xs = _split(lib, x, first[0] // 2) if M <= x_rows else None
    for n0 in range(0, N, w_rows):
        wn = w[n0:n0 + w_rows]
        ws = _split(lib, wn, 128)
        for m0 in range(0, M, x_rows):
            xm = x[m0:m0 + x_rows]
            m, n = xm.shape[0], wn.shape[0]
            bn, splits, whole = first if force or (m0 == 0 and n0 == 0) else plan(m, n, K, 0 if xs is None else first[0])
            xm_planes = xs if xs is not None else _split(lib, xm, bn // 2)
            whole = min(whole, -(-n // 256) - 1)
            partial = torch.empty(splits, m, n - 256 * whole, dtype=torch.float32, device=x.device) if splits > 1 else None
            b = bias[n0:n0 + n] if bias is not None else None
            ops._check(lib.mie_gemm_split(ops._ptr(xm_planes), ops._ptr(ws), ops._ptr(xm), ops._ptr(wn), ops._ptr(b),
                                          ops.tag(b) if b is not None else 0, ops._ptr(out[m0:m0 + m, n0:n0 + n]), ctypes.c_longlong(N),
                                          ops._ptr(partial), m, n, K, bn, splits, whole, ops._stream()), f"gemm_split M{m} N{n} K{K}")
    return out


def check_error() -> None:
    """Raises if a block gave up a bounded wait (call after a synchronise)."""
    lib = build._libs.get("gemm_split_tc")
    if lib is not None and lib.mie_gemm_split_error():
        lib.mie_gemm_split_clear_error()
        raise ops.KernelError("a block of the float32 tensor-core product gave up waiting on a barrier; its output is not valid")
