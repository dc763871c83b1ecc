"""What this library's users have it do, as cases that can be timed.

The work is LLM inference over quantized weights: single MUL_MAT calls from one activation column (decode) over small
batches to whole prompts (prefill), the projections of decode recorded in a CUDA graph, one layer's prefill and the
decode step of a model.  Shapes are those of the Qwen3-8B-shaped model that the repository's benchmark and decode harness
use (hidden 4096, 32 / 8 heads of 128, FFN 12288, vocabulary 151936); weights are seeded N(0, 0.02) in valid blocks,
packed on the device as a program packs them after loading; activations are N(0, 1).

A "mul_mat" case is one call of capi.mul_mat.  A "sweep" case replays a CUDA graph of a few layers' projections.  A
"layer" case runs one transformer layer over `m` prompt tokens behind `past` cached ones, op by op.  A "decode" case is
DecodeModel.run over `steps` tokens.
"""
import ctypes as C
import math

import torch

from scrapgpulibrary_b200 import capi
from scrapgpulibrary_b200.decode import DecodeConfig, DecodeModel

DTYPES = {"q4_0": 16, "q8_0": 17, "q4_k": 32, "q6_k": 33}
BLOCK = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_k": (256, 144), "q6_k": (256, 210)}
PACKED = 1
HIDDEN, HEADS, KV_HEADS, HEAD_DIM, FFN, VOCAB = 4096, 32, 8, 128, 12288, 151936
EPS = 1e-6


def listed():
    return [
        # the smallest call: one matvec over the joined Q, K and V rows of a layer, launch cost and latency count as much as bytes
        {"name": "matvec_q8_0", "kind": "mul_mat", "dtype": "q8_0", "k": 4096, "n": 6144, "m": 1},
        # the vocabulary head of a Q4_K_M model: one activation column over the largest matrix there is
        {"name": "head_q6_k", "kind": "mul_mat", "dtype": "q6_k", "k": 4096, "n": 151936, "m": 1},
        # the projections of decode, one column, as a program replays them: one graph over four layers' matrices
        {"name": "sweep_q4_k_m1", "kind": "sweep", "dtype": "q4_k", "layers": 4, "hidden": HIDDEN, "ffn": FFN, "m": 1},
        # the same for a few sequences decoded together, in the other K-quant of a Q4_K_M mix
        {"name": "sweep_q6_k_m4", "kind": "sweep", "dtype": "q6_k", "layers": 3, "hidden": HIDDEN, "ffn": FFN, "m": 4},
        # eight sequences decoded together, plain 4-bit weights
        {"name": "batch_q4_0_m8", "kind": "mul_mat", "dtype": "q4_0", "k": 4096, "n": 12288, "m": 8},
        # a batch between decode and prefill (parallel sequences, speculative tokens): the down projection for 24 columns
        {"name": "batch_q4_k_m24", "kind": "mul_mat", "dtype": "q4_k", "k": 12288, "n": 4096, "m": 24},
        # a short prompt, odd in every extent that may be odd
        {"name": "prompt_q4_0_m77", "kind": "mul_mat", "dtype": "q4_0", "k": 4096, "n": 5003, "m": 77},
        # a prompt of 512 tokens through the gate or up projection of an 8-bit model
        {"name": "prompt_q8_0_m512", "kind": "mul_mat", "dtype": "q8_0", "k": 4096, "n": 12288, "m": 512},
        # a long prompt through the same projection of a Q4_K model: the largest single product
        {"name": "prompt_q4_k_m2048", "kind": "mul_mat", "dtype": "q4_k", "k": 4096, "n": 12288, "m": 2048},
        # the down projection of the layers that a Q4_K_M mix keeps in Q6_K
        {"name": "prompt_q6_k_m512", "kind": "mul_mat", "dtype": "q6_k", "k": 12288, "n": 4096, "m": 512},
        # one layer of prefill behind an equally long cached prefix: norms, projections, rotation, cache stores, attention
        {"name": "layer_m512", "kind": "layer", "m": 512, "past": 512},
        # the decode step: six layers of the model and its full vocabulary head, four greedy tokens
        {"name": "decode", "kind": "decode", "layers": 6, "past": 1024, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges, in about the same proportions."""
    kind = rng.choice(["mul_mat"] * 8 + ["sweep"] * 2 + ["layer"] + ["decode"])
    if kind == "decode":
        return {"kind": "decode", "layers": rng.randint(2, 6), "past": rng.randint(64, 1100), "steps": rng.randint(1, 4)}
    if kind == "layer":
        return {"kind": "layer", "m": _log_int(rng, 48, 512), "past": rng.randint(0, 512)}
    if kind == "sweep":
        return {"kind": "sweep", "dtype": rng.choice(["q4_k", "q6_k"]), "layers": rng.randint(2, 4), "hidden": 256 * rng.randint(8, 20),
                "ffn": 256 * rng.randint(24, 56), "m": rng.choice([1, 1, 2, 3, 4, 5, 8])}
    dtype = rng.choice(sorted(DTYPES))
    lo, hi = rng.choice([(1, 1), (2, 8), (9, 32), (33, 160), (160, 1024)])
    m = _log_int(rng, lo, hi)
    k = 256 * _log_int(rng, 8, 48)
    n = _log_int(rng, 2048, 16384)
    if m == 1 and rng.random() < 0.3:
        n = _log_int(rng, 32000, VOCAB)
    if rng.random() < 0.7:
        n = max(64, n // 64 * 64)
    if m > 32:   # no more operations than the largest listed product of the format
        m = max(33, min(m, int(2.5e10 / (k * n))))
    return {"kind": "mul_mat", "dtype": dtype, "k": k, "n": n, "m": m}


# ---- inputs ------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _half_bytes(t):
    return t.to(torch.float16).contiguous().view(torch.uint8).reshape(t.shape + (2,))


def _ratio(a, b):
    return torch.where(b > 0, a / torch.where(b > 0, b, torch.ones_like(b)), torch.zeros_like(a))


def _blocks(dtype, w):
    """Natural GGUF blocks of f32 weights [n, k], with the absolute-maximum and min / max rules of synth.py."""
    n, k = w.shape
    if dtype == "q4_0":
        b = w.view(n, k // 32, 32)
        top = torch.gather(b, 2, b.abs().argmax(2, keepdim=True)).squeeze(2)
        d = top / -8.0
        inv = torch.where(d != 0, 1.0 / torch.where(d != 0, d, torch.ones_like(d)), torch.zeros_like(d))
        q = (b * inv[..., None] + 8.5).clamp(0, 15.99).to(torch.uint8)
        return torch.cat([_half_bytes(d), q[..., :16] | (q[..., 16:] << 4)], 2).view(n, -1)
    if dtype == "q8_0":
        b = w.view(n, k // 32, 32)
        d = b.abs().amax(2) / 127.0
        q = _ratio(b, d[..., None]).round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
        return torch.cat([_half_bytes(d), q], 2).view(n, -1)
    if dtype == "q4_k":
        b = w.view(n, k // 256, 8, 32)
        low = b.amin(3).clamp(max=0.0)
        scale, mins = (b.amax(3) - low) / 15.0, -low
        d, dmin = (scale.amax(2) / 63.0).half().float(), (mins.amax(2) / 63.0).half().float()
        ls = _ratio(scale, d[..., None]).round().clamp(0, 63).to(torch.uint8)
        lm = _ratio(mins, dmin[..., None]).round().clamp(0, 63).to(torch.uint8)
        ed, em = d[..., None] * ls, dmin[..., None] * lm
        q = _ratio(b + em[..., None], ed[..., None]).round().clamp(0, 15).to(torch.uint8).view(n, k // 256, 4, 2, 32)
        sc = torch.cat([ls[..., :4] | ((ls[..., 4:] >> 4) << 6), lm[..., :4] | ((lm[..., 4:] >> 4) << 6), (ls[..., 4:] & 15) | ((lm[..., 4:] & 15) << 4)], 2)
        qs = (q[..., 0, :] | (q[..., 1, :] << 4)).reshape(n, k // 256, 128)
        return torch.cat([_half_bytes(d), _half_bytes(dmin), sc, qs], 2).view(n, -1)
    b = w.view(n, k // 256, 16, 16)
    scale = b.abs().amax(3) / 31.0
    d = (scale.amax(2) / 127.0).half().float()
    sc = _ratio(scale, d[..., None]).round().clamp(0, 127).to(torch.int8)
    ed = d[..., None] * sc
    q = (_ratio(b, ed[..., None]).round().clamp(-32, 31) + 32).to(torch.uint8).view(n, k // 256, 2, 4, 32)
    ql = torch.cat([(q[..., 0, :] & 15) | ((q[..., 2, :] & 15) << 4), (q[..., 1, :] & 15) | ((q[..., 3, :] & 15) << 4)], 3).view(n, k // 256, 128)
    qh = ((q[..., 0, :] >> 4) | ((q[..., 1, :] >> 4) << 2) | ((q[..., 2, :] >> 4) << 4) | ((q[..., 3, :] >> 4) << 6)).view(n, k // 256, 64)
    return torch.cat([ql, qh, sc.view(torch.uint8), _half_bytes(d)], 2).view(n, -1)


def _natural(dtype, n, k, g):
    """uint8 [n, row bytes], made a few thousand rows at a time."""
    step = max(1, (1 << 25) // k)
    return torch.cat([_blocks(dtype, torch.randn(min(step, n - r), k, device="cuda", generator=g) * 0.02) for r in range(0, n, step)])


_stream = None


def _the_stream():
    """The program's one stream for single calls and graphs."""
    global _stream
    if _stream is None:
        torch.cuda.init()
        _stream = capi.Stream(0)
    return _stream


def _packed(dtype, n, k, g):
    nat = _natural(dtype, n, k, g)
    out = torch.empty(nat.numel(), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    s = _the_stream()
    capi.check(capi.lib().sm100_pack_device(s.handle, DTYPES[dtype], k, n, nat.data_ptr(), out.data_ptr()), "pack_device")
    s.sync()
    return out


def _shapes(case):
    """(k, n) of the projections of a sweep"""
    return (case["hidden"], case["hidden"]), (case["hidden"], case["ffn"]), (case["ffn"], case["hidden"])


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "mul_mat":
        k, n, m = case["k"], case["n"], case["m"]
        return {"case": case, "w": _packed(case["dtype"], n, k, g), "x": torch.randn(m, k, device="cuda", generator=g), "y": torch.empty(m, n, device="cuda")}
    if case["kind"] == "sweep":
        return _prepare_sweep(case, g)
    if case["kind"] == "layer":
        return _prepare_layer(case, g)
    return _prepare_decode(case, g)


def _prepare_sweep(case, g):
    s, m, dtype = _the_stream(), case["m"], case["dtype"]
    items = []
    for _ in range(case["layers"]):
        for k, n in _shapes(case):
            items.append((k, n, _packed(dtype, n, k, g), torch.randn(m, k, device="cuda", generator=g), torch.empty(m, n, device="cuda")))
    torch.cuda.synchronize()

    def enqueue():
        for k, n, w, x, y in items:
            capi.mul_mat(s, DTYPES[dtype], PACKED, w.data_ptr(), k, n, x.data_ptr(), m, y.data_ptr())

    enqueue()   # library scratch exists before the capture
    s.sync()
    graph = capi.Graph(s)
    with graph:
        enqueue()
    return {"case": case, "items": items, "graph": _GraphHandle(graph), "out": [i[4] for i in items]}


class _GraphHandle:
    """Destroys the graph with the state that owns it."""

    def __init__(self, graph):
        self.graph = graph

    def __del__(self):
        torch.cuda.synchronize()
        self.graph.destroy()


class _View(C.Structure):
    """sm100_view"""
    _fields_ = [("data", C.c_void_p), ("ne", C.c_int64 * 4), ("nb", C.c_int64 * 4)]

    def __init__(self, t, ne, strides):
        """strides in elements of 4 bytes"""
        super().__init__(t.data_ptr(), (C.c_int64 * 4)(*ne), (C.c_int64 * 4)(*[4 * v for v in strides]))


def _prepare_layer(case, g):
    """One more-bits layer of a Q4_K_M mix: attention value and FFN down projections in Q6_K, the rest in Q4_K."""
    m, past = case["m"], case["past"]
    ctx = past + m
    new = lambda *shape: torch.empty(*shape, device="cuda")   # noqa: E731
    w = {nm: (dt, k, n, _packed(dt, n, k, g)) for nm, dt, k, n in (
        ("q", "q4_k", HIDDEN, HEADS * HEAD_DIM), ("k", "q4_k", HIDDEN, KV_HEADS * HEAD_DIM), ("v", "q6_k", HIDDEN, KV_HEADS * HEAD_DIM),
        ("o", "q4_k", HEADS * HEAD_DIM, HIDDEN), ("gate", "q4_k", HIDDEN, FFN), ("up", "q4_k", HIDDEN, FFN), ("down", "q6_k", FFN, HIDDEN))}
    gain = {nm: 1.0 + 0.1 * torch.randn(n, device="cuda", generator=g) for nm, n in (("attn", HIDDEN), ("ffn", HIDDEN), ("q", HEAD_DIM), ("k", HEAD_DIM))}
    theta = torch.arange(ctx, device="cuda", dtype=torch.float64)[:, None] * (1e6 ** (-torch.arange(HEAD_DIM // 2, device="cuda", dtype=torch.float64) * 2 / HEAD_DIM))[None]
    st = {"case": case, "w": w, "gain": gain, "rope": torch.stack([theta.cos(), theta.sin()], 2).float().contiguous(),
          "pos": torch.arange(past, ctx, device="cuda", dtype=torch.int32),
          "x": torch.randn(m, HIDDEN, device="cuda", generator=g),
          "k_cache": torch.randn(KV_HEADS, ctx, HEAD_DIM, device="cuda", generator=g), "v_cache": torch.randn(KV_HEADS, ctx, HEAD_DIM, device="cuda", generator=g),
          "xn": new(m, HIDDEN), "q": new(m, HEADS, HEAD_DIM), "k": new(m, KV_HEADS, HEAD_DIM), "v": new(m, KV_HEADS, HEAD_DIM),
          "qh": new(HEADS, m, HEAD_DIM), "att": new(HEADS, m, HEAD_DIM), "merged": new(m, HEADS, HEAD_DIM),
          "proj": new(m, HIDDEN), "x1": new(m, HIDDEN), "gate": new(m, FFN), "up": new(m, FFN), "act": new(m, FFN), "y": new(m, HIDDEN), "x2": new(m, HIDDEN)}
    token_major = lambda t, heads: _View(t, (HEAD_DIM, m, heads, 1), (1, heads * HEAD_DIM, HEAD_DIM, heads * HEAD_DIM * m))   # noqa: E731
    head_major = lambda t, heads, rows: _View(t, (HEAD_DIM, rows, heads, 1), (1, HEAD_DIM, rows * HEAD_DIM, heads * rows * HEAD_DIM))   # noqa: E731
    st["views"] = {"q": token_major(st["q"], HEADS), "qh": head_major(st["qh"], HEADS, m), "k": token_major(st["k"], KV_HEADS), "v": token_major(st["v"], KV_HEADS),
                   "k_cache": head_major(st["k_cache"], KV_HEADS, ctx), "v_cache": head_major(st["v_cache"], KV_HEADS, ctx),
                   "att": head_major(st["att"], HEADS, m), "merged": token_major(st["merged"], HEADS), "pos": _View(st["pos"], (m, 1, 1, 1), (1, m, m, m))}
    return st


class _Weights:
    """The `weights` mapping of DecodeModel, one matrix at a time."""

    def __init__(self, cfg, seed):
        self.cfg, self.seed = cfg, seed
        c, sizes = cfg, {}
        for i in range(c.layers):
            v = "q6_k" if c.more_bits(i) else "q4_k"
            for nm, dt, n, k in (("wq", "q4_k", c.heads * c.head_dim, c.hidden), ("wk", "q4_k", c.kv_heads * c.head_dim, c.hidden), ("wv", v, c.kv_heads * c.head_dim, c.hidden),
                                 ("wo", "q4_k", c.hidden, c.heads * c.head_dim), ("wgate", "q4_k", c.ffn, c.hidden), ("wup", "q4_k", c.ffn, c.hidden), ("wdown", v, c.hidden, c.ffn)):
                sizes["l%d.%s" % (i, nm)] = (dt, n, k)
        sizes["embed"], sizes["head"] = ("q4_k", c.vocab, c.hidden), ("q6_k", c.vocab, c.hidden)
        self.sizes = sizes
        self.vectors = {"l%d.%s" % (i, nm): n for i in range(c.layers)
                        for nm, n in (("attn_norm", c.hidden), ("ffn_norm", c.hidden), ("q_norm", c.head_dim), ("k_norm", c.head_dim))}
        self.vectors["out_norm"] = c.hidden

    def __contains__(self, name):
        return name in self.sizes or name in self.vectors

    def __getitem__(self, name):
        g = _gen(self.seed * 1000 + sorted(list(self.sizes) + list(self.vectors)).index(name))
        if name in self.vectors:
            return (1.0 + 0.1 * torch.randn(self.vectors[name], device="cuda", generator=g)).cpu().numpy()
        dt, n, k = self.sizes[name]
        return DTYPES[dt], _natural(dt, n, k, g).cpu().numpy(), k


def _prepare_decode(case, g):
    past = case["past"]
    cfg = DecodeConfig(layers=case["layers"], start_pos=past, n_ctx=past + 32)
    model = DecodeModel(cfg, weights=_Weights(cfg, int(torch.randint(1 << 30, (1,), device="cuda", generator=g))))
    first = torch.randint(VOCAB, (1,), device="cuda", generator=g, dtype=torch.int32)
    model.reset(0)
    model.capture()
    for lw in model.layers:
        for nm in ("k_cache", "v_cache"):
            lw[nm].zero_()
            lw[nm][:, :past].normal_(generator=g)
    torch.cuda.synchronize()
    out = {"logits": model.logits, "tokens": model.tokens_out[:case["steps"]], "k": [lw["k_cache"] for lw in model.layers], "v": [lw["v_cache"] for lw in model.layers]}
    return {"case": case, "model": model, "first": first, "out": out}


# ---- one pass ----------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "mul_mat":
        capi.mul_mat(_stream, DTYPES[case["dtype"]], PACKED, state["w"].data_ptr(), case["k"], case["n"], state["x"].data_ptr(), case["m"], state["y"].data_ptr())
        return state["y"]
    if case["kind"] == "sweep":
        state["graph"].graph.launch()
        return state["out"]
    if case["kind"] == "layer":
        return _run_layer(state)
    model, here = state["model"], torch.cuda.current_stream()
    model.tstream.wait_stream(here)
    with torch.cuda.stream(model.tstream):
        model.token.copy_(state["first"])
        model.pos.fill_(case["past"])
        model.step_index.zero_()
    model.run(case["steps"])
    here.wait_stream(model.tstream)
    return state["out"]


def _run_layer(st):
    L, s, v, m, past = capi.lib(), _stream.handle, st["views"], st["case"]["m"], st["case"]["past"]
    ctx = past + m
    p = lambda nm: C.c_void_p(st[nm].data_ptr())   # noqa: E731
    gain = lambda nm: C.c_void_p(st["gain"][nm].data_ptr())   # noqa: E731
    ok = capi.check

    def mm(name, x, y):
        dt, k, n, w = st["w"][name]
        capi.mul_mat(_stream, DTYPES[dt], PACKED, w.data_ptr(), k, n, st[x].data_ptr(), m, st[y].data_ptr())

    ok(L.sm100_rms_norm(s, p("x"), None, gain("attn"), None, p("xn"), HIDDEN, m, EPS))
    mm("q", "xn", "q")
    mm("k", "xn", "k")
    mm("v", "xn", "v")
    ok(L.sm100_rms_norm(s, p("q"), None, gain("q"), None, p("q"), HEAD_DIM, HEADS * m, EPS))
    ok(L.sm100_rms_norm(s, p("k"), None, gain("k"), None, p("k"), HEAD_DIM, KV_HEADS * m, EPS))
    ok(L.sm100_rope(s, p("q"), p("pos"), p("rope"), 0, ctx, p("q"), HEAD_DIM, HEADS, m, HEAD_DIM, 1))
    ok(L.sm100_rope(s, p("k"), p("pos"), p("rope"), 0, ctx, p("k"), HEAD_DIM, KV_HEADS, m, HEAD_DIM, 1))
    ok(L.sm100_set_rows_view(s, C.byref(v["k"]), 0, C.byref(v["pos"]), 0, C.byref(v["k_cache"]), 0))
    ok(L.sm100_set_rows_view(s, C.byref(v["v"]), 0, C.byref(v["pos"]), 0, C.byref(v["v_cache"]), 0))
    ok(L.sm100_cpy(s, C.byref(v["q"]), 0, C.byref(v["qh"]), 0))
    ok(L.sm100_attention(s, p("qh"), p("k_cache"), p("v_cache"), None, 1, p("att"), HEAD_DIM, HEAD_DIM, m, ctx, HEADS, KV_HEADS, 1, past, None, HEAD_DIM ** -0.5))
    ok(L.sm100_cpy(s, C.byref(v["att"]), 0, C.byref(v["merged"]), 0))
    mm("o", "merged", "proj")
    ok(L.sm100_rms_norm(s, p("x"), p("proj"), gain("ffn"), p("x1"), p("xn"), HIDDEN, m, EPS))
    mm("gate", "xn", "gate")
    mm("up", "xn", "up")
    ok(L.sm100_swiglu(s, p("gate"), p("up"), p("act"), m * FFN))
    mm("down", "act", "y")
    ok(L.sm100_add(s, p("x1"), p("y"), p("x2"), m * HIDDEN))
    return {"x": st["x2"], "k": st["k_cache"], "v": st["v_cache"]}


# ---- what a pass cannot do without -------------------------------------------------------------------

def _weight_bytes(dtype, n, k):
    be, bb = BLOCK[dtype]
    return n * k // be * bb


def _product(dtype, n, k, m):
    return {"bytes": _weight_bytes(dtype, n, k) + 4 * k * m + 4 * n * m, "flops": 2 * n * k * m}


def _layer_products(more_bits, m):
    dt = "q6_k" if more_bits else "q4_k"
    return [_product("q4_k", HEADS * HEAD_DIM, HIDDEN, m), _product("q4_k", KV_HEADS * HEAD_DIM, HIDDEN, m), _product(dt, KV_HEADS * HEAD_DIM, HIDDEN, m),
            _product("q4_k", HIDDEN, HEADS * HEAD_DIM, m), _product("q4_k", FFN, HIDDEN, m), _product("q4_k", FFN, HIDDEN, m), _product(dt, HIDDEN, FFN, m)]


def work(case):
    if case["kind"] == "mul_mat":
        return _product(case["dtype"], case["n"], case["k"], case["m"])
    if case["kind"] == "sweep":
        parts = [_product(case["dtype"], n, k, case["m"]) for k, n in _shapes(case)] * case["layers"]
        return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
    kv_row = 2 * 4 * KV_HEADS * HEAD_DIM
    if case["kind"] == "layer":
        m, past = case["m"], case["past"]
        w = sum(_weight_bytes(dt, n, k) for dt, k, n in (("q4_k", HIDDEN, 5120), ("q6_k", HIDDEN, 1024), ("q4_k", HIDDEN, HIDDEN), ("q4_k", HIDDEN, 2 * FFN), ("q6_k", FFN, HIDDEN)))
        pairs = m * past + m * (m + 1) // 2
        # the residual in and out, the cached prefix read, the new rows written
        return {"bytes": w + 2 * 4 * m * HIDDEN + kv_row * (past + m), "flops": sum(p["flops"] for p in _layer_products(True, m)) + 4 * HEADS * HEAD_DIM * pairs}
    c = DecodeConfig(layers=case["layers"])
    bytes_, flops = 0, 0
    for i in range(case["steps"]):
        for layer in range(c.layers):
            for p in _layer_products(c.more_bits(layer), 1):
                bytes_, flops = bytes_ + p["bytes"], flops + p["flops"]
        vis = case["past"] + i + 1
        head = _product("q6_k", VOCAB, HIDDEN, 1)
        bytes_ += c.layers * kv_row * vis + head["bytes"]
        flops += c.layers * 4 * HEADS * HEAD_DIM * vis + head["flops"]
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the error against a float64 evaluation.  Up to 32 columns, and with Q6_K at any number, the library
    multiplies 16-bit integer activations with the exact weights (2e-5 to 5e-5); wider batches of the other formats multiply f16
    roundings of both (3e-4, Q4_K 7e-4), and a layer holds such products (1e-3)."""
    if case["kind"] == "mul_mat" and case["m"] > 32 and case["dtype"] != "q6_k":
        return {"rel": 3e-3 if case["dtype"] == "q4_k" else 1.2e-3}
    if case["kind"] in ("mul_mat", "sweep"):
        return {"rel": 2e-4}
    return {"rel": 4e-3} if case["kind"] == "layer" else {"rel": 2e-3, "differ": 0.0}
