"""What a user of the engine has it do, as cases that can be timed and checked: whole steps of a Llama model, and single layers of
the designs that the engine serves, each called through the public step function or through the part registry.

A case is a dict of plain values.  ``part`` says what runs, ``size`` its sizes (the presets' and the benchmark's), ``dtype`` the
mode, and the rest the step's batch: ``portions`` prompt portions with ``new`` tokens between them, every other one on top of
``earlier`` positions, and ``decoding`` requests with one new token each, the longest of them on ``context`` positions.

Steps of decoded tokens alone, and a step that is one prompt of a whole model, run from a captured CUDA graph, as the engine runs them; everything else
is launched call by call, as the engine launches mixed steps."""
import math
import random

import numpy as np
import torch

from mini_inference_engine_b200.cache.storage import CacheLayout, CacheStorage
from mini_inference_engine_b200.config import PartSpec, load_preset
from mini_inference_engine_b200.engine.batch import BatchBuilder, BatchRow
from mini_inference_engine_b200.models import DecoderModel
from mini_inference_engine_b200.parts import Runtime, build_part

DEV = "cuda"
PAGE = 16
TAPS = 4
EPS = 1e-5
UNIT_EPS = 1e-6
GATE_CAP = 15.0
EXPERTS, TOP = 16, 4

# TinyLlama-1.1B, Llama-3-8B, and the two layer sizes of the benchmark's design comparison
SIZES = {
    "tinyllama": dict(width=2048, ff=5632, heads=32, kv_heads=4, dim=64, theta=10000.0, layers=22, vocab=32000, positions=2048),
    "llama-8b": dict(width=4096, ff=14336, heads=32, kv_heads=8, dim=128, theta=500000.0, positions=8192),
    "w2048": dict(width=2048, heads=16, ret_heads=8, dim=128, expert_ff=2112),
    "w4096": dict(width=4096, heads=32, ret_heads=16, dim=128, expert_ff=5376),
}
RECURRENT = ("retention", "channel_delta", "head_delta", "matrix_memory")


def _case(part, size, dtype="bf16", portions=0, new=0, earlier=0, decoding=0, context=0, name=None):
    c = dict(part=part, size=size, dtype=dtype, portions=portions, new=new, earlier=earlier, decoding=decoding, context=context)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # one decode step of a whole model serving eight users: the benchmark's headline workload
        _case("model", "tinyllama", decoding=8, context=512, name="model-decode-8"),
        # a long prompt through the whole model: the time to the first token, and the benchmark's prefill figure
        _case("model", "tinyllama", portions=1, new=2048, name="model-prompt-2048"),
        # one layer's attention while 64 users decode at contexts of 1,024 to 4,096: the long serving workload
        _case("attention", "llama-8b", decoding=64, context=4096, name="attention-decode-64"),
        # chunked prefill: two ragged portions in a step, one of them continuing a prompt
        _case("attention", "llama-8b", portions=2, new=1937, earlier=1500, name="attention-prompt-ragged"),
        # the feed-forward of a single user's decode step: the smallest call, all latency
        _case("feed_forward", "tinyllama", decoding=1, context=512, name="feed-forward-decode-1"),
        # the true 32-bit mode (verification of a checkpoint, reference logits): a medium prompt
        _case("feed_forward", "tinyllama", "fp32", portions=1, new=509, name="feed-forward-prompt-fp32"),
        _case("attention", "tinyllama", "fp32", portions=2, new=1000, earlier=300, name="attention-prompt-fp32"),
        # linear attention with a fixed decay, 32 users decoding
        _case("retention", "w2048", decoding=32, context=700, name="retention-decode-32"),
        # the gated delta rule with a decay per key channel over two prompts of unequal length
        _case("channel_delta", "w2048", portions=2, new=1500, name="channel-delta-prompt"),
        # the gated delta rule with a decay per head: a prompt portion beside decoding users, the continuous-batching step
        _case("head_delta", "w2048", portions=1, new=1500, decoding=16, context=900, name="head-delta-mixed"),
        # a matrix memory with exponential gates over one long prompt
        _case("matrix_memory", "w2048", portions=1, new=2048, name="matrix-memory-prompt"),
        # routed experts (four of sixteen) over a prompt portion
        _case("experts", "w2048", portions=1, new=1024, name="experts-prompt"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    part = rng.choice(["model", "attention", "attention", "feed_forward", "feed_forward", "retention", "channel_delta", "head_delta",
                       "matrix_memory", "experts"])
    decode = rng.random() < 0.4
    if part == "model":
        size, dtype = "tinyllama", "bf16"
    elif part in ("attention", "feed_forward"):
        size = rng.choice(["tinyllama", "llama-8b"])
        dtype = "fp32" if rng.random() < 0.4 else "bf16"
        if dtype == "fp32":
            size = "tinyllama"
    else:
        size, dtype = rng.choice(["w2048", "w2048", "w4096"]), "bf16"
    if decode:
        return _case(part, size, dtype, decoding=_log(rng, 1, 64), context=_log(rng, 32, 2000))
    most = 1024 if dtype == "fp32" else 2048
    portions = 1 if part in ("model", "feed_forward", "experts") else rng.randint(1, 3)
    new = max(_log(rng, 40, most), 2 * portions)
    earlier = rng.choice([0, _log(rng, 30, 900)]) if part in ("attention",) + RECURRENT else 0
    decoding = rng.choice([0, _log(rng, 1, 32)]) if part in ("attention",) + RECURRENT else 0
    return _case(part, size, dtype, portions=portions, new=new, earlier=earlier, decoding=decoding, context=_log(rng, 32, 1500) if decoding else 0)


# --------------------------------------------------------------------------- the batch and its inputs

def rows_of(case):
    """[(new tokens, earlier positions)] of the step's rows."""
    P, R = case["portions"], case["decoding"]
    rows, left = [], case["new"]
    for i in range(P):
        n = left if i == P - 1 else max(1, case["new"] * (i + 1) * 2 // (P * (P + 1)))
        rows.append((n, case["earlier"] if i % 2 == 0 else 0))
        left -= n
    for j in range(R):
        ctx = case["context"] - (j * (3 * case["context"] // 4)) // max(1, R - 1)
        rows.append((1, max(1, ctx - 1)))
    return rows


def _dtype(case):
    return torch.float32 if case["dtype"] == "fp32" else torch.bfloat16


def _gen(seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 7919 + sum(ord(ch) * 257 ** (i % 5) for i, ch in enumerate(what))) % (1 << 62))
    return g


def _normal(seed, what, shape, std=1.0, mean=0.0):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(mean, std, generator=_gen(seed, what))


def _uniform(seed, what, shape, lo, hi):
    return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=_gen(seed, what))


def weights(case, seed):
    """The checkpoint's tensors, stored in 16 bits as checkpoints are (the 32-bit mode widens them)."""
    s = SIZES[case["size"]]
    w = s["width"]
    out = {}

    def normal(name, *shape, std=None, mean=0.0):
        out[name] = _normal(seed, name, shape, shape[-1] ** -0.5 if std is None else std, mean).to(torch.bfloat16)

    def uniform(name, lo, hi, *shape):
        out[name] = _uniform(seed, name, shape, lo, hi).to(torch.bfloat16)

    def llama_attention(p):
        normal(p + "q_proj.weight", s["heads"] * s["dim"], w, std=0.02)
        normal(p + "k_proj.weight", s["kv_heads"] * s["dim"], w, std=0.02)
        normal(p + "v_proj.weight", s["kv_heads"] * s["dim"], w, std=0.02)
        normal(p + "o_proj.weight", w, s["heads"] * s["dim"], std=0.02)

    def llama_mlp(p):
        normal(p + "gate_proj.weight", s["ff"], w, std=0.02)
        normal(p + "up_proj.weight", s["ff"], w, std=0.02)
        normal(p + "down_proj.weight", w, s["ff"], std=0.02)

    part = case["part"]
    if part == "model":
        normal("model.embed_tokens.weight", s["vocab"], w, std=0.02)
        for i in range(s["layers"]):
            p = f"model.layers.{i}."
            llama_attention(p + "self_attn.")
            llama_mlp(p + "mlp.")
            normal(p + "input_layernorm.weight", w, std=0.1, mean=1.0)
            normal(p + "post_attention_layernorm.weight", w, std=0.1, mean=1.0)
        normal("model.norm.weight", w, std=0.1, mean=1.0)
        normal("lm_head.weight", s["vocab"], w, std=0.02)
    elif part == "attention":
        llama_attention("")
    elif part == "feed_forward":
        llama_mlp("")
    elif part == "retention":
        H, D, V = s["ret_heads"], 128, 256
        for n, rows in (("q", H * D), ("k", H * D), ("v", H * V), ("g", H * V)):
            normal(n, rows, w)
        normal("o", w, H * V)
    elif part == "matrix_memory":
        H, D, V = s["ret_heads"], 128, 256
        for n, rows in (("q", H * D), ("k", H * D), ("v", H * V), ("g", H * V), ("i", H), ("f", H)):
            normal(n, rows, w)
        normal("o", w, H * V)
        normal("norm", H * V, std=0.1, mean=1.0)
        normal("i.b", H, std=1.0)
        normal("f.b", H, std=1.0, mean=3.0)
    elif part in ("channel_delta", "head_delta"):
        H, D = s["heads"], s["dim"]
        G = H if part == "channel_delta" else H // 2
        for n, rows in (("q", G * D), ("k", G * D), ("v", H * D)):
            normal(n, rows, w)
            normal(n + ".conv", rows, TAPS, std=0.5)
        normal("b", H, w)
        uniform("A_log", -3.0, 0.5, H)
        normal("norm", D, std=0.1, mean=1.0)
        if part == "channel_delta":
            r = w // 16
            normal("a1", r, w)
            normal("a2", H * D, r)
            normal("g1", r, w)
            normal("g2", H * D, r)
            uniform("dt_bias", -4.0, 1.0, H * D)
        else:
            normal("a", H, w)
            normal("g", H * D, w)
            uniform("dt_bias", -4.0, 1.0, H)
        normal("o", w, H * D)
    elif part == "experts":
        normal("router", EXPERTS, w)
        for e in range(EXPERTS):
            normal(f"e{e}.up", s["expert_ff"], w)
            normal(f"e{e}.down", w, s["expert_ff"])
    return out


def states(case, seed):
    """What the requests' state slots hold before the step (slot r + 1 is row r's; a request's first portion starts from zeros)."""
    part, s = case["part"], SIZES[case["size"]]
    rows = rows_of(case)
    if part == "retention":
        shapes = [(s["ret_heads"], 256, 128)]
    elif part == "matrix_memory":
        shapes = [(s["ret_heads"], 257, 128), (s["ret_heads"],)]
    elif part in ("channel_delta", "head_delta"):
        H, D = s["heads"], s["dim"]
        C = (3 if part == "channel_delta" else 2) * H * D
        shapes = [(H, D, D), (TAPS - 1 if part == "channel_delta" else TAPS, C)]
    else:
        return []
    out = []
    for i, sh in enumerate(shapes):
        t = _normal(seed, f"state{i}", (len(rows) + 1,) + sh, 1.0 if i else 0.3)
        if part == "matrix_memory" and i == 1:
            t = t.abs()                                     # a running maximum that started at zero
        t[0] = 0
        for r, (_, earlier) in enumerate(rows):
            if earlier == 0:
                t[r + 1] = 0
        out.append(t)
    return out


def _tables(case, seed):
    """Every row's block table: pages handed out in the order a pool in use gives them, page 0 left for padding."""
    rows = rows_of(case)
    counts = [-(-(n + e) // PAGE) for n, e in rows]
    ids = list(range(1, sum(counts) + 1))
    random.Random(int(seed) + 17).shuffle(ids)
    tables, at = [], 0
    for c in counts:
        tables.append(np.array(ids[at:at + c], dtype=np.int32))
        at += c
    return tables, sum(counts) + 1


def _pages(case, seed, pages, layer):
    """Keys and values of the earlier positions (and whatever the other pages held): [2, pages, key heads, PAGE, dim]."""
    s = SIZES[case["size"]]
    return _normal(seed, f"pages{layer}", (2, pages, s["kv_heads"], PAGE, s["dim"]), 0.9).to(_dtype(case))


def _inputs(case, seed):
    """The layer's input, a normed stream: [tokens, width]."""
    T = sum(n for n, _ in rows_of(case))
    return _normal(seed, "x", (T, SIZES[case["size"]]["width"])).to(torch.bfloat16)


def _tokens(case, seed):
    r = np.random.RandomState((int(seed) * 31 + 5) % (1 << 31))
    return [r.randint(0, SIZES[case["size"]]["vocab"], n).astype(np.int32) for n, _ in rows_of(case)]


def _ret_decay(H):
    return [1.0 - 2.0 ** (-5 - i % 8) for i in range(H)]


def _part(case):
    s, part = SIZES[case["size"]], case["part"]
    w = s["width"]
    if part == "attention":
        return build_part("mixer", PartSpec("attention", dict(
            hidden_size=w, num_heads=s["heads"], num_kv_heads=s["kv_heads"], head_dim=s["dim"],
            position=PartSpec("rope", dict(head_dim=s["dim"], rotary_dim=s["dim"], theta=s["theta"], max_position=s["positions"])))))
    if part == "feed_forward":
        return build_part("feed_forward", PartSpec("swiglu", dict(hidden_size=w, intermediate_size=s["ff"])))
    if part == "retention":
        return build_part("mixer", PartSpec("retention", dict(hidden_size=w, num_heads=s["ret_heads"], dim=128, vdim=256, decay=_ret_decay(s["ret_heads"]),
                                                              rot_dims=128, rot_base=1e4, eps=EPS)))
    if part == "matrix_memory":
        return build_part("mixer", PartSpec("matrix_memory", dict(hidden_size=w, num_heads=s["ret_heads"], dim=128, vdim=256, eps=EPS, gate_cap=GATE_CAP)))
    if part == "channel_delta":
        return build_part("mixer", PartSpec("channel_delta", dict(hidden_size=w, num_heads=s["heads"], num_kv_heads=s["heads"], dim=s["dim"], vdim=s["dim"],
                                                                  taps=TAPS, eps=EPS, decay_rank=w // 16, gate_rank=w // 16, unit_eps=UNIT_EPS)))
    if part == "head_delta":
        return build_part("mixer", PartSpec("head_delta", dict(hidden_size=w, num_heads=s["heads"], num_kv_heads=s["heads"] // 2, dim=s["dim"], vdim=s["dim"],
                                                               taps=TAPS, eps=EPS, unit_eps=UNIT_EPS)))
    if part == "experts":
        return build_part("feed_forward", PartSpec("routed_experts", dict(hidden_size=w, num_experts=EXPERTS, top=TOP, expert_size=s["expert_ff"])))
    raise ValueError(part)


# --------------------------------------------------------------------------- one case

class State:
    pass


@torch.inference_mode()
def prepare(case, seed):
    st = State()
    rows = rows_of(case)
    rt = Runtime(DEV, _dtype(case))
    tables, pages = _tables(case, seed)
    W = weights(case, seed)
    whole = case["part"] == "model"
    if whole:
        model = DecoderModel(load_preset(case["size"] + "-1.1b").model_spec(), W, rt)
        storage = model.allocate_cache(pages, PAGE, len(rows))
        layout = model.cache_layout
    else:
        part = _part(case)
        part.bind(W, rt)
        layout = CacheLayout.from_needs({0: part.cache_need() if hasattr(part, "cache_need") else None})
        storage = CacheStorage(layout, pages, PAGE, len(rows), rt.dtype, DEV)
    del W
    tokens = _tokens(case, seed) if whole else [np.zeros(n, dtype=np.int32) for n, _ in rows]
    batch = [BatchRow(t, e, [tab] * len(layout.groups), r + 1, (n - 1,)) for r, ((n, e), t, tab) in enumerate(zip(rows, tokens, tables))]
    ctx = BatchBuilder(len(layout.groups), PAGE, DEV, SIZES[case["size"]].get("positions")).build(batch)
    out = {}
    if whole:
        def forward():
            out["logits"] = model.step(ctx)
    else:
        x = _inputs(case, seed).to(rt.dtype)
        if hasattr(part, "cache_need"):
            cache = storage.layer_cache(0)

            def forward():
                out["out"] = part.forward(x, ctx, cache)
        else:
            def forward():
                out["out"] = part.forward(x, ctx)
    st.graph = None
    # requests whose first tokens these are: the engine clears their state slots in front of the step
    st.fresh = [r + 1 for r, (_, e) in enumerate(rows) if e == 0] if case["part"] in RECURRENT else []
    if case["portions"] == 0 or whole:
        for layer, t in storage.kv.items():
            t.zero_()
        forward()
        torch.cuda.synchronize()
        st.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st.graph):
            forward()
    for layer, t in storage.kv.items():
        t.copy_(_pages(case, seed, pages, layer))
    for key, value in zip(sorted(storage.state, key=str), states(case, seed)):
        storage.state[key].copy_(value)
    if case["part"] == "attention":
        out["pages"] = storage.kv[0]
    for i, key in enumerate(sorted(storage.state, key=str)):
        out[f"state{i}"] = storage.state[key]
    st.out, st.forward, st.storage = out, forward, storage
    torch.cuda.synchronize()
    return st


@torch.inference_mode()
def run(state):
    if state.graph is not None:
        state.graph.replay()
    else:
        for slot in state.fresh:
            state.storage.clear_state_slot(slot)
        state.forward()
    return dict(state.out)


# --------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    s, rows, part = SIZES[case["size"]], rows_of(case), case["part"]
    w = s["width"]
    T = sum(n for n, _ in rows)
    el = 4 if case["dtype"] == "fp32" else 2

    def attention(h):
        params = w * (h["heads"] + 2 * h["kv_heads"]) * h["dim"] + w * h["heads"] * h["dim"]
        seen = sum(n * e + n * (n + 1) // 2 for n, e in rows)
        kv = 2 * h["kv_heads"] * h["dim"] * el
        return params, params * 2 * T + 4 * h["heads"] * h["dim"] * seen, kv * sum(n + e for n, e in rows)

    if part == "model":
        a, fl, kv = attention(s)
        mlp = 3 * w * s["ff"]
        W = len(rows)
        return {"bytes": 2 * (s["layers"] * (a + mlp) + s["vocab"] * w) + s["layers"] * kv + 2 * T * w + 4 * W * s["vocab"],
                "flops": s["layers"] * (fl + 2 * T * mlp) + 2 * W * s["vocab"] * w}
    if part == "attention":
        a, fl, kv = attention(s)
        return {"bytes": el * (a + 2 * T * w) + kv, "flops": fl}
    if part == "feed_forward":
        return {"bytes": el * (3 * w * s["ff"] + 2 * T * w), "flops": 6 * T * w * s["ff"]}
    if part == "experts":
        E = min(EXPERTS, T * TOP)
        return {"bytes": 2 * 2 * E * w * s["expert_ff"] + 4 * EXPERTS * w + T * w * 6, "flops": 4 * T * TOP * w * s["expert_ff"]}
    R = len(rows)
    if part in ("retention", "matrix_memory"):
        H, D, V = s["ret_heads"], 128, 256
        params, state = w * H * (2 * D + 2 * V) + w * H * V, H * D * V
        recurrence = 4 * state
    else:
        H, D = s["heads"], s["dim"]
        G = H if part == "channel_delta" else H // 2
        params, state = w * (2 * G + 2 * H) * D + w * H * D, H * D * D
        if part == "channel_delta":
            params = w * (2 * G + H) * D + w * H * D + 2 * (w // 16) * (w + H * D)
        recurrence = 6 * state
    return {"bytes": 2 * params + 2 * T * w + 4 * T * w + 8 * R * state, "flops": T * (2 * params + recurrence)}


# Four times what two right implementations were seen to differ by (or the error of the start against 64 bits, where that is more telling):
# one 16-bit rounding is 4e-3 of a value and 2e-3 in the mean, and a layer has two to five in a row; 32-bit sums differ by 1e-6.
def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["part"] == "model":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 1e-2, "max": 0.2}


# --------------------------------------------------------------------------- the same in 64 bits, in plain torch

def _rotate(x, pos, freq):
    """Rotate-half over the last dimension; the angle (position times frequency) is a 32-bit number by definition."""
    angle = (pos.float()[:, None] * freq.float()[None, :]).double()
    c, sn = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    h = x.shape[-1] // 2
    a, b = x[..., :h], x[..., h:]
    return torch.cat([a * c - b * sn, b * c + a * sn], -1)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _llama_attention(x, W, p, s, rows, tables, pages):
    """x [tokens, width] -> (output, pages with the new keys and values), all 64-bit."""
    H, G, D = s["heads"], s["kv_heads"], s["dim"]
    lin = lambda t, n: t @ W[p + n + ".weight"].double().t()
    j = torch.arange(0, D, 2, dtype=torch.int64).float()
    freq = (1.0 / (s["theta"] ** (j / D))).to(DEV)
    out = torch.empty(x.shape[0], H * D, dtype=torch.float64, device=DEV)
    at = 0
    for (n, e), table in zip(rows, tables):
        pos = torch.arange(e, e + n, device=DEV)
        xr = x[at:at + n]
        q = _rotate(lin(xr, "q_proj").view(n, H, D), pos, freq)
        k = _rotate(lin(xr, "k_proj").view(n, G, D), pos, freq)
        v = lin(xr, "v_proj").view(n, G, D)
        t = torch.from_numpy(table.astype(np.int64)).to(DEV)
        pages[0][t[pos // PAGE], :, pos % PAGE] = k
        pages[1][t[pos // PAGE], :, pos % PAGE] = v
        flat = lambda i: pages[i][t].permute(1, 0, 2, 3).reshape(G, -1, D)[:, :e + n]
        K, V = flat(0), flat(1)
        for g in range(G):
            qs = q[:, g * (H // G):(g + 1) * (H // G)].permute(1, 0, 2)
            sc = qs @ K[g].t() * D ** -0.5
            sc = sc.masked_fill(torch.arange(e + n, device=DEV)[None, :] > pos[:, None], -math.inf)
            o = torch.softmax(sc, -1) @ V[g]
            out[at:at + n].view(n, H, D)[:, g * (H // G):(g + 1) * (H // G)] = o.permute(1, 0, 2)
        at += n
    return lin(out, "o_proj"), pages


def _llama_mlp(x, W, p):
    lin = lambda t, n: t @ W[p + n + ".weight"].double().t()
    return lin(torch.nn.functional.silu(lin(x, "gate_proj")) * lin(x, "up_proj"), "down_proj")


def _conv_silu(x, before, taps):
    """x [n, C] after the taps - 1 inputs ``before`` (oldest first); taps [C, TAPS], the last one for the newest input."""
    ext = torch.cat([before, x], 0)
    y = sum(ext[i:i + x.shape[0]] * taps[:, i] for i in range(TAPS))
    return torch.nn.functional.silu(y)


@torch.inference_mode()
def exact(case, seed):
    part, s, rows = case["part"], SIZES[case["size"]], rows_of(case)
    W = weights(case, seed)
    tables, pages = _tables(case, seed)
    if part == "model":
        ids = torch.from_numpy(np.concatenate(_tokens(case, seed)).astype(np.int64)).to(DEV)
        res = W["model.embed_tokens.weight"][ids].double()
        norm = lambda t, n: _rms(t, EPS) * W[n].double()
        for i in range(s["layers"]):
            p = f"model.layers.{i}."
            a, _ = _llama_attention(norm(res, p + "input_layernorm.weight"), W, p + "self_attn.", s, rows, tables,
                                    _pages(case, seed, pages, i).double())
            res = res + a
            res = res + _llama_mlp(norm(res, p + "post_attention_layernorm.weight"), W, p + "mlp.")
        last = torch.tensor(np.cumsum([n for n, _ in rows]) - 1, device=DEV)
        return {"logits": norm(res[last], "model.norm.weight") @ W["lm_head.weight"].double().t()}
    x = _inputs(case, seed).double()
    if part == "attention":
        out, kv = _llama_attention(x, W, "", s, rows, tables, _pages(case, seed, pages, 0).double())
        return {"out": out, "pages": kv}
    if part == "feed_forward":
        return {"out": _llama_mlp(x, W, "")}
    W = {n: t.double() for n, t in W.items()}
    if part == "experts":
        z = x @ W["router"].t()
        val, idx = torch.topk(z, TOP, dim=-1)
        wt = torch.softmax(val, -1)
        out = torch.zeros_like(x)
        for e in range(EXPERTS):
            t, j = (idx == e).nonzero(as_tuple=True)
            out[t] += wt[t, j][:, None] * (torch.relu(x[t] @ W[f"e{e}.up"].t()) ** 2 @ W[f"e{e}.down"].t())
        return {"out": out}
    before = [t.double() for t in states(case, seed)]
    outs, at = [], 0
    for r, (n, e) in enumerate(rows):
        S = before[0][r + 1]                                                       # [heads, vdim, dim]
        xr = x[at:at + n]
        at += n
        pos = torch.arange(e, e + n, device=DEV)
        if part == "retention":
            H, D, V = s["ret_heads"], 128, 256
            freq = torch.tensor([1e4 ** (-2.0 * i / D) for i in range(D // 2)], dtype=torch.float32, device=DEV)
            q = _rotate((xr @ W["q"].t()).view(n, H, D), pos, freq)
            k = _rotate((xr @ W["k"].t()).view(n, H, D), pos, freq) * D ** -0.5
            v = (xr @ W["v"].t()).view(n, H, V)
            keep = torch.tensor(_ret_decay(H), dtype=torch.float32, device=DEV).double()[None].expand(n, H)
            o = torch.empty(n, H, V, dtype=torch.float64, device=DEV)
            for t in range(n):
                S = keep[t][:, None, None] * S + v[t][:, :, None] * k[t][:, None, :]
                o[t] = (S * q[t][:, None, :]).sum(-1)
            o = _rms(o, EPS).reshape(n, H * V)
            outs.append((o * torch.nn.functional.silu(xr @ W["g"].t())) @ W["o"].t())
            before[0][r + 1] = S
        elif part == "matrix_memory":
            H, D, V = s["ret_heads"], 128, 256
            q = (xr @ W["q"].t()).view(n, H, D) * D ** -0.5
            k = (xr @ W["k"].t()).view(n, H, D)
            v = torch.cat([(xr @ W["v"].t()).view(n, H, V), torch.ones(n, H, 1, dtype=torch.float64, device=DEV)], -1)
            cap = lambda z: GATE_CAP * torch.tanh(z / GATE_CAP)
            gi, gf = cap(xr @ W["i"].t() + W["i.b"]), torch.nn.functional.logsigmoid(cap(xr @ W["f"].t() + W["f.b"]))
            m = before[1][r + 1]
            o = torch.empty(n, H, V, dtype=torch.float64, device=DEV)
            for t in range(n):
                new = torch.maximum(gf[t] + m, gi[t])
                keep, write = torch.exp(gf[t] + m - new), torch.exp(gi[t] - new)
                S = keep[:, None, None] * S + v[t][:, :, None] * (write[:, None] * k[t])[:, None, :]
                m = new
                y = (S * q[t][:, None, :]).sum(-1)
                o[t] = y[:, :V] / (torch.maximum(y[:, V].abs(), torch.exp(-m)) + 1e-6)[:, None]
            o = _rms(o, EPS).reshape(n, H * V) * W["norm"] * torch.sigmoid(xr @ W["g"].t())
            outs.append(o @ W["o"].t())
            before[0][r + 1], before[1][r + 1] = S, m
        else:
            H, D = s["heads"], s["dim"]
            G = H if part == "channel_delta" else H // 2
            old = before[1][r + 1]
            if part == "head_delta":                        # a ring: the input of position p lies in row p % TAPS
                old = torch.stack([old[(e - i) % TAPS] for i in range(TAPS - 1, 0, -1)])
            proj = xr @ torch.cat([W["q"], W["k"], W["v"]], 0).t()
            taps = torch.cat([W["q.conv"], W["k.conv"], W["v.conv"]], 0)
            y = _conv_silu(proj, old, taps)
            unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + UNIT_EPS)
            q = (unit(y[:, :G * D].reshape(n, G, D)) * D ** -0.5).repeat_interleave(H // G, 1)
            k = unit(y[:, G * D:2 * G * D].reshape(n, G, D)).repeat_interleave(H // G, 1)
            v = y[:, 2 * G * D:].reshape(n, H, D)
            beta = torch.sigmoid(xr @ W["b"].t())
            A = torch.exp(W["A_log"])
            if part == "channel_delta":
                dt = torch.nn.functional.softplus(xr @ W["a1"].t() @ W["a2"].t() + W["dt_bias"]).view(n, H, D)
                keep = torch.exp(-A[None, :, None] * dt)
                gate = torch.sigmoid(xr @ W["g1"].t() @ W["g2"].t())
            else:
                keep = torch.exp(-A * torch.nn.functional.softplus(xr @ W["a"].t() + W["dt_bias"]))[:, :, None].expand(n, H, D)
                gate = torch.nn.functional.silu(xr @ W["g"].t())
            o = torch.empty(n, H, D, dtype=torch.float64, device=DEV)
            for t in range(n):
                S = keep[t][:, None, :] * S
                u = beta[t][:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
                S = S + u[:, :, None] * k[t][:, None, :]
                o[t] = (S * q[t][:, None, :]).sum(-1)
            o = (_rms(o, EPS) * W["norm"]).reshape(n, H * D) * gate
            outs.append(o @ W["o"].t())
            before[0][r + 1] = S
            ext = torch.cat([old, proj], 0)
            if part == "channel_delta":
                before[1][r + 1] = ext[-(TAPS - 1):]
            else:
                for i in range(min(TAPS - 1, n)):           # (a portion leaves what the next token's taps reach)
                    before[1][r + 1][(e + n - 1 - i) % TAPS] = proj[n - 1 - i]
    got = {"out": torch.cat(outs)}
    got.update({f"state{i}": t for i, t in enumerate(before)})
    return got
