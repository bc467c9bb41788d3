"""Chooses the attention kernels for a step.

float32 (the true 32-bit path): tiles of (token, head) pairs whose products run on the tensor cores with every operand as three
bfloat16 parts (``csrc/attention_f32.cu``, heads of up to 128) for rows with many new tokens and, on long contexts, for rows of a few and
of one; a warp a pair on the CUDA cores (``csrc/attention_simt.cu``) for the rest.
bfloat16: rows with one new token go to the tensor-core decode kernel (context split across
blocks), rows with more go to a prefill kernel -- the tcgen05 one for head sizes 64 and 128, the
mma.sync one for the other multiples of 16 up to 128; head sizes beyond those kernels fall back to
the CUDA-core kernel, which takes every size up to 256.  ``set_backend("simt")`` forces the CUDA-core
kernel everywhere (used by tests to compare the two)."""
from __future__ import annotations

import torch

from . import ops
from .device import num_sms

_backend = "auto"
_prefill_backend = "tcgen05"


def set_prefill_backend(name: str) -> None:
    global _prefill_backend
    if name not in ("tcgen05", "mma"):
        raise ValueError(name)
    _prefill_backend = name


def set_backend(name: str) -> None:
    global _backend
    if name not in ("auto", "simt"):
        raise ValueError(name)
    _backend = name


def _row_kinds(ctx) -> tuple:
    """(rows of one token, rows of more, tokens of those) of the step, or None where the host does not know the rows'
    lengths (a captured step).  Counted once a step, not once a layer: a step may hold hundreds of rows."""
    kinds = ctx.host.get("_row_kinds", False)
    if kinds is False:
        q_lens = ctx.host.get("q_len")
        kinds = None
        if q_lens is not None:
            long = [n for n in q_lens if n > 1]
            kinds = (len(q_lens) - len(long), len(long), sum(long))
        ctx.host["_row_kinds"] = kinds
    return kinds


def decode_only(ctx) -> bool:
    """Whether every row of the step has exactly one new token (known on the host)."""
    kinds = _row_kinds(ctx)
    return kinds is not None and kinds[1] == 0 and kinds[0] > 0


def rotates_in_decode(dtype, head_dim: int, ctx) -> bool:
    """Whether ``attention(..., rope=...)`` can rotate q and the new key itself and write the cache: a step of
    decoding rows only, on the tensor-core decode kernel, with a head size it rotates."""
    return (_backend == "auto" and dtype == torch.bfloat16 and head_dim <= 128 and head_dim % 32 == 0
            and decode_only(ctx))


# float32: tiles of (token, head) pairs (csrc/attention_f32.cu) against a warp a pair.  A tile takes as long with one pair as with 64, a walk of keys shared out over up to eight
# blocks some 15 us a thousand positions; a warp takes 120 us for them, and warps fill the GPU from about 1,500 pairs on.  One row, us, a warp a pair : tiles, 0 / 250 / 500 / 1,000 /
# 2,000 earlier positions -- 32 heads of 64 on 4: 2 tokens 6 : 10 / 33 : 13 / 64 : 19 / 125 : 19 / 244 : 33, 32 tokens 7 : 10 / 42 : 20 / 76 : 26 / 146 : 28 / 282 : 43, 64 tokens
# 13.4 : 10.7 / 74 : 21 / 122 : 28 / 222 : 35 / 426 : 50; 16 of 64 on 16: 32 tokens 7 : 10 / 40 : 20 / 73 : 26 / 138 : 29 / 266 : 39; 32 of 128 on 8: 32 tokens 8 : 19 / 55 : 24 / 100 : 35 / 192 : 48 /
# 372 : 60.  R rows of one token on 250 / 1,000 / 4,000 positions: 32 of 64 on 4, R 1 33 : 12 / 125 : 19 / 481 : 59, 16 36 : 17 / 134 : 47 / 604 : 171, 64 77 : 45 / 304 : 169 / 1,181 : 656;
# 16 of 64 on 16, 4 30 : 16 / 111 : 47 / 515 : 170, 16 35 : 44 / 148 : 166 / 566 : 644; 32 of 128 on 8, 1 38 : 19 / 143 : 32 / 555 : 107, 4 38 : 20 / 144 : 44, 16 48 : 67 / 217 : 245.
F32_MIN_WORK = 1536         # (token, head) pairs of the rows that tiles could take, from which they do ...
F32_MIN_WORK_FRESH = 2048   # ... where no row has more than F32_FRESH positions; any number of pairs ...
F32_FRESH = 256
F32_LONG = 640              # ... where a row reaches this many positions: rows of one token too where tiles are faster (F32_FULL_GROUP, F32_FEW)
F32_LONG_STEP = 128         # the same for a step of rows of one token only
F32_WIDE_WORK = 135_000     # heads above 64: pairs times positions for every round of tiles up to which warps take less (32 heads of 128 on 8, us, a warp a pair : tiles -- 64 tokens
                            # alone 17 : 20, 64 on 30 23 : 26, two rows of 40 18 : 20, four 27 : 20; 16 of 96 on 16, 16 rows of 20 tokens 20 : 23, 32 33 : 47, 16 rows of 40 40 : 25)
F32_MIN_PAIRS = 16          # pairs of a row on one key head below which it is left to the warps: three quarters of its tile would be empty
F32_FULL_GROUP = 8          # query heads on a key head from which a row of one token fills enough of a tile (heads of up to 64) ...
F32_FEW = 64                # ... or so few such (row, key head) pairs that their tiles run side by side


def captured_context_bounds(dtype) -> tuple:
    """Context bounds, beside the longest one, that a captured step is worth planning for: the choice of kernel above goes by the bound, since a captured step's positions change.
    float32, few rows: planned for 960 positions or more a row of one token takes a tile, some 12 us on 10 positions too, where a warp a pair takes 6 (32 heads of 64 on 4);
    a portion of 32 tokens 14 against 7."""
    return (F32_LONG_STEP - 1,) if dtype == torch.float32 else ()


def _attention_f32(args, ctx, out, num_heads, num_kv_heads, head_dim, page_size, scale, window, mods, keep):
    """float32: rows with at least F32_MIN_PAIRS (token, head of a group) pairs by tiles, shorter ones one pair a warp, as all are in a step of few
    pairs on few positions; on many positions rows of any length by tiles.  Where the host does not know the rows' lengths (a captured step) each of the two kernels takes the
    rows that are its own."""
    group = num_heads // num_kv_heads
    min_q_len = max(2, -(-F32_MIN_PAIRS // group))
    q_lens = ctx.host.get("q_len")
    reach = ctx.max_ctx_len if window == 0 else min(ctx.max_ctx_len, abs(window) + keep)
    singles = ctx.row_q_len.numel() if q_lens is None else q_lens.count(1) if isinstance(q_lens, list) else int((q_lens == 1).sum())
    if ((reach >= F32_LONG or (reach >= F32_LONG_STEP and decode_only(ctx)))
            and ((group >= F32_FULL_GROUP and head_dim <= 64) or singles * num_kv_heads <= F32_FEW)):
        min_q_len = 1
    long = None if q_lens is None else [n for n in q_lens if n >= min_q_len]
    longest, c_lens = ctx.max_ctx_len, ctx.host.get("ctx_len")
    if long and len(long) < len(q_lens) and c_lens is not None and len(c_lens) == len(q_lens) and max(c_lens) == longest:
        # the rows that tiles would take, not those beside them, decide (captured steps are planned for more than the host's numbers say).  Us, 20 tokens on 50 positions of 16 heads of
        # 64 on 16 beside 8 rows of one token on 700: a launch of tiles for that portion alone 99, all rows by warps 82
        longest = max(c for n, c in zip(q_lens, c_lens) if n >= min_q_len)
        reach = longest if window == 0 else min(longest, abs(window) + keep)
    sizes = (ctx.num_tokens, out, num_heads, num_kv_heads, head_dim, page_size, scale, window)
    pairs = (ctx.num_tokens if long is None else sum(long)) * num_heads
    few = F32_MIN_WORK_FRESH if longest <= F32_FRESH else F32_MIN_WORK if reach < F32_LONG else 1
    if head_dim > 64 and long and min_q_len > 1 and reach < F32_LONG:
        rounds = sum(-(-n * group // 128) for n in long) * num_kv_heads / num_sms()
        few = max(few, F32_WIDE_WORK * max(1.0, rounds) / longest)
    if pairs < few and min_q_len > 1:
        return ops.paged_attention(*args, *sizes, mods=mods, keep=keep)
    if min_q_len > 1 and (long is None or len(long) < len(q_lens)):
        ops.paged_attention(*args, *sizes, mods=mods, keep=keep, below=min_q_len)
    ops.attention_f32(*args, *sizes, min_q_len=min_q_len, mods=mods, keep=keep, work=None if long is None else (len(long), sum(long)), max_ctx=longest)
    return out


def attention(qkv, ctx, cache, out, num_heads, num_kv_heads, head_dim, scale, window, rope=None, q_stride=None, mods=None,
              keep: int = 0):
    """``rope`` = (cos, sin): ``qkv`` is unrotated and the cache rows of the new tokens are unwritten; only
    where ``rotates_in_decode`` holds.  ``window``: None or 0 all earlier keys, w > 0 the last w positions, w < 0 the
    keys of the query's own block of -w positions.  ``keep``: beside a window or block, the first ``keep`` keys of the
    sequence stay in sight.  ``q_stride``: elements between the token rows of ``qkv`` (by
    default rows of a fused q|k|v projection).  ``mods`` (``ops.ScoreMods``): a cap on the scores, a bias or a slope by distance, a sink in
    the softmax; every kernel applies them (the tcgen05 kernel for portions in an instance of its own)."""
    if q_stride is None:
        q_stride = (num_heads + 2 * num_kv_heads) * head_dim
    args = (qkv, q_stride, cache.k, cache.v, ctx.block_tables[cache.group], ctx.row_q_start, ctx.row_q_len,
            ctx.row_ctx_len)
    fast = _backend == "auto" and qkv.dtype == torch.bfloat16 and head_dim <= 128
    window = int(window or 0)
    # the keys a single new token can reach, for the decode kernel's plan: a window or a block of positions bounds them
    keep = int(keep or 0) if window else 0              # (without a window every key is in sight already)
    reach = ctx.max_ctx_len if window == 0 else min(ctx.max_ctx_len, abs(window) + 64 + -(-keep // 64) * 64)
    if rope is not None:
        if mods is not None or keep:
            raise ValueError("rotation inside attention does not go together with score modifiers or kept keys")
        if not rotates_in_decode(qkv.dtype, head_dim, ctx):
            raise ValueError("rotation inside attention serves steps of decoding rows only (bfloat16, head sizes "
                             "in steps of 32 up to 128)")
        return ops.decode_attention(*args, out, num_heads, num_kv_heads, head_dim, cache.page_size, scale, window,
                                    max_ctx=ctx.max_ctx_len, rope=rope)
    if not fast and _backend == "auto" and ops.attention_f32_takes(qkv, cache.k, cache.v, out, head_dim):
        return _attention_f32(args, ctx, out, num_heads, num_kv_heads, head_dim, cache.page_size, scale, window, mods, keep)
    if not fast:
        return ops.paged_attention(*args, ctx.num_tokens, out, num_heads, num_kv_heads, head_dim, cache.page_size,
                                   scale, window, mods=mods, keep=keep)
    kinds = _row_kinds(ctx)
    has_decode = kinds is None or kinds[0] > 0
    has_prefill = kinds is None or kinds[1] > 0
    min_q_len = 2
    if kinds is None and ctx.host.get("few_single_rows"):
        # row lengths unknown here (a captured step), but rows of one token are the exception among them: the
        # kernel for portions takes those too, and the launch of the decode kernel is saved
        has_decode, min_q_len = False, 1
    if has_decode:
        ops.decode_attention(*args, out, num_heads, num_kv_heads, head_dim, cache.page_size, scale, window,
                             max_ctx=reach, mods=mods, keep=keep)
    if has_prefill:
        # tcgen05 (S and O in tensor memory) for the head sizes it is written for, mma.sync otherwise
        # (combinations of kept keys and score modifiers that the tcgen05 kernel has no instance for: mma.sync)
        tc = (head_dim in (64, 128) and cache.page_size >= 8 and q_stride % 8 == 0 and _prefill_backend == "tcgen05"
              and (mods is None or mods.tcgen05_takes(keep)))
        fn = ops.prefill_attention_tc if tc else ops.prefill_attention
        # the rows that are portions, and their tokens: the launch is laid out for those, not for every decoding row
        work = None if kinds is None else (kinds[1], kinds[2])
        fn(*args, ctx.num_tokens, out, num_heads, num_kv_heads, head_dim, cache.page_size, scale, window,
           min_q_len=min_q_len, work=work, mods=mods, keep=keep)
    return out
