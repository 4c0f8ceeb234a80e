"""Timed cases: the work a serving program has this library do, through its public entry points.

Four kinds of pass cover it:

  step      one decode step of a few decoder layers (`decode_step.decode_step`): the token loop of a server;
  attend    new keys and values into the paged cache, then attention over it: decode (one query row per
            request) and prefill (a chunk of a prompt behind what is already cached), int8 or fp32 pools;
  linear    one projection on its own: int4 group-wise, asymmetric int4, weight-only int8, W8A8 with the
            activations quantised per token on the way, fp8 with one scale per tensor; from one row
            (a single stream) to a full prefill batch.  With few rows a pass walks several weight
            matrices, as a token walks the layers of a model;
  quantize  loading a model: weights into (or out of) their storage format.

Widths, head counts, groups and lengths are those of this repository's benchmark and tests, or generic
multiples around them; row counts and context lengths are ragged, as requests are.
"""
from __future__ import annotations

import math

import torch

import longhornai_b200 as lb
from longhornai_b200 import decode_step as ds

HEAD_DIM, PAGE = 128, 16


def listed():
    return [
        # A single stream of a chat program, launched eagerly: the smallest step, where every launch shows.
        {"name": "step one stream", "kind": "step", "batch": 1, "ctx": 777, "ragged": False, "layers": 4, "dim": 4096,
         "n_q": 32, "n_kv": 8, "ffn": 14336, "graph": False},
        # A server's full decode batch with 2048 tokens of context each, replayed as a CUDA graph.
        {"name": "step batch 32", "kind": "step", "batch": 32, "ctx": 2048, "ragged": False, "layers": 4, "dim": 4096,
         "n_q": 32, "n_kv": 8, "ffn": 14336, "graph": True},
        # One request through the single-request calls: a program that drives sequences one at a time.
        {"name": "attend one request", "kind": "attend", "pool": "int8", "n_req": 1, "seq_q": 1, "ctx": 1234, "n_q": 32,
         "n_kv": 8, "window": 0},
        # A large decode batch of ragged contexts, 512 to 4096 tokens: the attention of a busy server.
        {"name": "attend batch 64", "kind": "attend", "pool": "int8", "n_req": 64, "seq_q": 1, "ctx": 4096, "n_q": 32,
         "n_kv": 8, "window": 0},
        # A chunk of a long prompt: 1000 new tokens behind 3000 cached ones.
        {"name": "attend prompt chunk", "kind": "attend", "pool": "int8", "n_req": 1, "seq_q": 1000, "ctx": 4000, "n_q": 32,
         "n_kv": 8, "window": 0},
        # A small decode batch over an unquantised cache.
        {"name": "attend fp32 batch 8", "kind": "attend", "pool": "fp32", "n_req": 8, "seq_q": 1, "ctx": 2048, "n_q": 32,
         "n_kv": 8, "window": 0},
        # The MLP up-projection of eight layers for one token: the int4 decode GEMV.
        {"name": "int4 one row", "kind": "linear", "fmt": "w4", "M": 1, "K": 4096, "N": 14336, "group": 128, "mats": 8},
        # The same projection for the prompt tokens of a prefill chunk.
        {"name": "int4 prefill", "kind": "linear", "fmt": "w4", "M": 1000, "K": 4096, "N": 14336, "group": 128, "mats": 1},
        # Weight-only int8 for a small batch.
        {"name": "int8 16 rows", "kind": "linear", "fmt": "w8", "M": 16, "K": 4096, "N": 4096, "group": 0, "mats": 8},
        # W8A8 at the largest prefill shape, activations quantised per token in the pass.
        {"name": "W8A8 prefill 8192", "kind": "linear", "fmt": "w8a8", "M": 8192, "K": 8192, "N": 28672, "group": 0, "mats": 1},
        # fp8 for a short ragged prompt.
        {"name": "fp8 prompt 333", "kind": "linear", "fmt": "fp8", "M": 333, "K": 4096, "N": 14336, "group": 0, "mats": 1},
        # Loading: one MLP projection into int4 groups.
        {"name": "load int4", "kind": "quantize", "fmt": "w4", "rows": 4096, "cols": 14336, "group": 128, "back": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi, unit):
    return max(unit, unit * round(_log(rng, lo, hi) / unit))


def draw(rng):
    kind = rng.choice(["step", "attend", "attend", "linear", "linear", "linear", "quantize"])
    if kind == "step":
        dim, n_q, n_kv, ffn = rng.choice([(4096, 32, 8, 14336), (4096, 32, 8, 14336), (1024, 8, 2, 3584), (2048, 16, 8, 5632)])
        return {"kind": "step", "batch": _log(rng, 1, 32), "ctx": _log(rng, 32, 2048), "ragged": rng.random() < 0.5,
                "layers": rng.randint(2, 4), "dim": dim, "n_q": n_q, "n_kv": n_kv, "ffn": ffn, "graph": rng.random() < 0.5}
    if kind == "attend":
        n_q, n_kv = rng.choice([(32, 8), (32, 8), (64, 8), (16, 16), (8, 2)])
        form = rng.choice(["one", "batch", "batch", "chunk", "fp32"])
        window = rng.choice([0, 0, 0, _log(rng, 128, 2048)])
        if form == "one":
            return {"kind": "attend", "pool": "int8", "n_req": 1, "seq_q": 1, "ctx": _log(rng, 16, 4096), "n_q": n_q,
                    "n_kv": n_kv, "window": window}
        if form == "batch":
            return {"kind": "attend", "pool": "int8", "n_req": _log(rng, 2, 64), "seq_q": 1, "ctx": _log(rng, 64, 4096),
                    "n_q": n_q, "n_kv": n_kv, "window": window}
        if form == "chunk":
            new = _log(rng, 8, 1000)
            return {"kind": "attend", "pool": "int8", "n_req": 1, "seq_q": new, "ctx": new + rng.choice([0, rng.randint(1, 3000)]),
                    "n_q": min(n_q, 32), "n_kv": n_kv, "window": window}
        return {"kind": "attend", "pool": "fp32", "n_req": _log(rng, 1, 8), "seq_q": 1, "ctx": _log(rng, 64, 2048),
                "n_q": n_q, "n_kv": n_kv, "window": window}
    if kind == "linear":
        fmt = rng.choice(["w4", "w4", "w4a", "w8", "w8a8", "fp8"])
        rows = {"w4": 1000, "w4a": 1000, "w8": 512, "w8a8": 4096, "fp8": 2048}[fmt]
        M = _log(rng, 1, rows)
        group = {"w4": rng.choice([128, 128, 64, 32]), "w4a": 128}.get(fmt, 0)
        K = _width(rng, 1024, 4096 if fmt in ("w4", "w4a", "w8") else 8192, 128)
        return {"kind": "linear", "fmt": fmt, "M": M, "K": K, "N": _width(rng, 1024, 14336, 16), "group": group,
                "mats": 8 if M <= 64 else 1}
    return {"kind": "quantize", "fmt": rng.choice(["w4", "w4a", "w8", "w8row", "fp8"]), "rows": _width(rng, 1024, 4096, 128),
            "cols": _width(rng, 1024, 14336, 16), "group": 128, "back": rng.random() < 0.3}


# ---- inputs ----------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(g, K, N):
    return torch.randn(K, N, device="cuda", generator=g).mul_(0.02)


def _lengths(g, n, ctx, ragged):
    """Cached tokens of each request after this pass: all `ctx`, or uniform from an eighth of it."""
    if not ragged:
        return [ctx] * n
    lo = max(1, ctx // 8)
    return torch.randint(lo, ctx + 1, (n,), device="cuda", generator=g).tolist()


def _tables(g, lens, longest):
    """Block tables with room for the `longest` request over a shuffled pool that could hold as many of it;
    unused entries -1."""
    blocks = [-(-n // PAGE) for n in lens]
    width = -(-longest // PAGE)
    pool = len(lens) * width
    perm = torch.randperm(pool, device="cuda", generator=g).to(torch.int32)
    t = torch.full((len(lens), width), -1, dtype=torch.int32, device="cuda")
    used = 0
    for r, b in enumerate(blocks):
        t[r, :b] = perm[used:used + b]
        used += b
    return t, pool


def _fill(g, pools, tables, lens, L):
    """Cached tokens of every request, through the cache's own append."""
    for r, n in enumerate(lens):
        if n <= 0:
            continue
        k = torch.randn(L.n_kv_heads, n, L.head_dim, device="cuda", generator=g)
        v = torch.randn(L.n_kv_heads, n, L.head_dim, device="cuda", generator=g)
        (lb.paged_kv_append_q8 if len(pools) == 4 else lb.paged_kv_append)(*pools, k, v, tables[r], L, 0, n)


def _prepare_step(c, g):
    cfg = ds.StepConfig(c["dim"], c["n_q"], c["n_kv"], HEAD_DIM, c["ffn"])
    lens = _lengths(g, c["batch"], c["ctx"], c["ragged"])
    tables, pool = _tables(g, [n + 1 for n in lens], c["ctx"] + 1)
    L = lb.PagedLayout(pool, PAGE, c["n_kv"], HEAD_DIM)
    acfg = lb.PagedAttnCfg(c["n_q"], c["n_kv"], 1, HEAD_DIM, 1, 0.0, 0, 0)
    layers, pools = [], []
    for _ in range(c["layers"]):
        gain = lambda: 1.0 + 0.1 * torch.randn(c["dim"], device="cuda", generator=g)  # noqa: E731
        w = lambda k, n: _weights(g, k, n)  # noqa: E731
        layers.append(ds.LayerWeights.quantize(cfg, w(cfg.dim, cfg.q_dim), w(cfg.dim, cfg.kv_dim), w(cfg.dim, cfg.kv_dim),
                                               w(cfg.q_dim, cfg.dim), w(cfg.dim, 2 * cfg.ffn), w(cfg.ffn, cfg.dim), gain(), gain()))
        kv = ds.KVPools.empty(L, "cuda")
        _fill(g, (kv.k, kv.v, kv.ks, kv.vs), tables, lens, L)
        pools.append(kv)
    past = torch.tensor(lens, dtype=torch.int32, device="cuda")
    emb = torch.randn(c["batch"], cfg.dim, device="cuda", generator=g)
    s = {"emb": emb, "x": torch.empty_like(emb), "layers": layers, "pools": pools, "tables": tables, "past": past,
         "cur": past + 1, "cfg": cfg, "L": L, "acfg": acfg, "buf": ds.StepBuffers.allocate(cfg, c["batch"], emb.device)}
    if c["graph"]:                       # one eager step, then the capture that a server keeps
        _step(s)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _step(s)
    return s


def _step(s):
    s["x"].copy_(s["emb"])               # the tokens' embeddings enter the residual stream
    ds.decode_step(s["x"], s["layers"], s["pools"], s["tables"], s["past"], s["cur"], s["cfg"], s["L"], s["acfg"], s["buf"])


def _prepare_attend(c, g):
    new = c["seq_q"]
    lens = _lengths(g, c["n_req"], c["ctx"], c["n_req"] > 1)
    past = [n - new for n in lens]
    tables, pool = _tables(g, lens, c["ctx"])
    L = lb.PagedLayout(pool, PAGE, c["n_kv"], HEAD_DIM)
    shape = (pool, c["n_kv"], PAGE, HEAD_DIM)
    if c["pool"] == "int8":
        pools = tuple(torch.zeros(shape, dtype=torch.int8, device="cuda") for _ in range(2)) + \
            tuple(torch.zeros(shape[:3], device="cuda") for _ in range(2))
        _fill(g, pools, tables, past, L)
    else:
        pools = tuple(torch.zeros(shape, device="cuda") for _ in range(2))
        _fill(g, pools, tables, lens, L)
    rnd = lambda *dims: torch.randn(*dims, device="cuda", generator=g)  # noqa: E731
    n = c["n_req"]
    q = rnd(c["n_q"], new, HEAD_DIM) if n == 1 and c["pool"] == "int8" else rnd(n, c["n_q"], new, HEAD_DIM)
    kv = (c["n_kv"], new, HEAD_DIM) if n == 1 else (n, c["n_kv"], new, HEAD_DIM)
    return {"q": q, "k": rnd(*kv), "v": rnd(*kv), "pools": pools, "tables": tables, "table": tables[0], "o": torch.empty_like(q),
            "past": torch.tensor(past, dtype=torch.int32, device="cuda"), "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"),
            "past0": past[0], "len0": lens[0], "L": L,
            "acfg": lb.PagedAttnCfg(c["n_q"], c["n_kv"], new, HEAD_DIM, 1, 0.0, c["window"], 0)}


QUANT = {
    "w4": lambda w, c: lb.q4_quantize_groupwise(w, c["group"]),
    "w4a": lambda w, c: lb.q4a_quantize_groupwise(w, c["group"]),
    "w8": lambda w, c: lb.q8_quantize_per_col(w),
    "w8a8": lambda w, c: lb.q8_quantize_per_col(w),
    "w8row": lambda w, c: lb.q8_quantize_per_row(w),
    "fp8": lambda w, c: lb.fp8_quantize_per_tensor(w),
}
DEQUANT = {
    "w4": lambda q, c: lb.q4_dequantize_groupwise(*q, c["group"]),
    "w4a": lambda q, c: lb.q4a_dequantize_groupwise(*q, c["group"]),
    "w8": lambda q, c: lb.q8_dequantize_per_col(*q),
    "w8row": lambda q, c: lb.q8_dequantize_per_row(*q),
    "fp8": lambda q, c: lb.fp8_dequantize(*q, 0),
}


def prepare(case, seed):
    c, g = case, _gen(seed)
    if c["kind"] == "step":
        s = _prepare_step(c, g)
    elif c["kind"] == "attend":
        s = _prepare_attend(c, g)
    elif c["kind"] == "linear":
        mats = [QUANT[c["fmt"]](_weights(g, c["K"], c["N"]), c) for _ in range(c["mats"])]
        if c["fmt"] == "fp8":            # the weight's scale is known when the model is loaded
            mats = [(q, float(sc.item())) for q, sc in mats]
        xs = [torch.randn(c["M"], c["K"], device="cuda", generator=g).bfloat16().float() for _ in mats]
        s = {"mats": mats, "xs": xs}
    else:
        w = _weights(g, c["rows"], c["cols"])
        s = {"w": QUANT[c["fmt"]](w, c) if c["back"] else w}
    s["case"] = c
    return s


# ---- one pass -----------------------------------------------------------------------------------------

def _attend(c, s):
    if c["pool"] == "fp32":
        return lb.paged_attention_batched_f32(s["q"], *s["pools"], s["tables"], s["lens"], s["acfg"], s["L"], O=s["o"])
    if c["n_req"] == 1:
        lb.paged_kv_append_q8(*s["pools"], s["k"], s["v"], s["table"], s["L"], s["past0"], c["seq_q"])
        o = lb.paged_attention_q8(s["q"], *s["pools"], s["table"], s["len0"], s["acfg"], s["L"], O=s["o"])
    else:
        lb.paged_kv_append_q8_batched(*s["pools"], s["k"], s["v"], s["tables"], s["past"], s["L"], 1)
        o = lb.paged_attention_q8_batched(s["q"], *s["pools"], s["tables"], s["lens"], s["acfg"], s["L"], O=s["o"])
    return [o, *s["pools"]]


def _linear(c, x, m):
    if c["fmt"] == "w4":
        return lb.gemm_w4a16_groupwise(x, *m, c["group"])
    if c["fmt"] == "w4a":
        return lb.gemm_w4a16_asym(x, *m, c["group"])
    if c["fmt"] == "w8":
        return lb.gemm_w8a16_perchannel(x, *m)
    if c["fmt"] == "w8a8":
        xq, xs = lb.q8_quantize_per_row(x)
        return lb.gemm_w8a8(xq, m[0], xs, m[1])
    xq, xs = lb.fp8_quantize_per_tensor(x)
    return lb.gemm_fp8_e4m3(xq, m[0], float(xs.item()), m[1])


def run(state):
    c = state["case"]
    if c["kind"] == "step":
        if c["graph"]:
            state["graph"].replay()
        else:
            _step(state)
        return [state["x"]] + [t for kv in state["pools"] for t in (kv.k, kv.v, kv.ks, kv.vs)]
    if c["kind"] == "attend":
        return _attend(c, state)
    if c["kind"] == "linear":
        return [_linear(c, x, m) for x, m in zip(state["xs"], state["mats"])]
    return DEQUANT[c["fmt"]](state["w"], c) if c["back"] else QUANT[c["fmt"]](state["w"], c)


# ---- what a pass cannot do without -----------------------------------------------------------------------

def _weight_bytes(fmt, K, N, group):
    if fmt in ("w4", "w4a"):
        return K * N / 2 + 4 * (K // group) * N
    return K * N + (4 * N if fmt in ("w8", "w8a8") else 4 * K if fmt == "w8row" else 4)


def _mean_len(c):
    """Expected cached tokens of a request."""
    ragged = c["ragged"] if c["kind"] == "step" else c["n_req"] > 1
    return (max(1, c["ctx"] // 8) + c["ctx"]) / 2 if ragged else float(c["ctx"])


def work(case):
    c = case
    if c["kind"] == "step":
        q, kv = c["n_q"] * HEAD_DIM, c["n_kv"] * HEAD_DIM
        mats = [(c["dim"], q + 2 * kv), (q, c["dim"]), (c["dim"], 2 * c["ffn"]), (c["ffn"], c["dim"])]
        tokens = c["batch"] * (_mean_len(c) + 1)
        return {"bytes": c["layers"] * (sum(_weight_bytes("w4", k, n, 128) for k, n in mats) + tokens * c["n_kv"] * (2 * HEAD_DIM + 8)
                                        + 8 * c["dim"]) + 8 * c["batch"] * c["dim"],
                "flops": c["layers"] * (2.0 * c["batch"] * sum(k * n for k, n in mats) + 4.0 * tokens * q)}
    if c["kind"] == "attend":
        new, n = c["seq_q"], c["n_req"]
        length = _mean_len(c)
        window = c["window"] or length
        seen = sum(min(length - new + i + 1, window) for i in range(new))        # keys of the query rows of one request
        keys = min(length, window + new - 1)
        row = 2 * HEAD_DIM + 8 if c["pool"] == "int8" else 8 * HEAD_DIM
        append = n * new * c["n_kv"] * (8 * HEAD_DIM + row) if c["pool"] == "int8" else 0
        return {"bytes": n * keys * c["n_kv"] * row + append + 8 * n * new * c["n_q"] * HEAD_DIM,
                "flops": 4.0 * n * seen * c["n_q"] * HEAD_DIM}
    if c["kind"] == "linear":
        return {"bytes": c["mats"] * (_weight_bytes(c["fmt"], c["K"], c["N"], c["group"]) + 4 * c["M"] * (c["K"] + c["N"])),
                "flops": c["mats"] * 2.0 * c["M"] * c["K"] * c["N"]}
    return {"bytes": 4 * c["rows"] * c["cols"] + _weight_bytes(c["fmt"], c["rows"], c["cols"], c["group"]), "flops": 0}


def tolerance(case):
    c = case
    if c["kind"] == "quantize" or c.get("fmt") == "w8a8":
        return "exact"                   # integer sums and codes, one rounding each
    if c["kind"] == "step":
        # up to four layers of chained fp32 operators; a cache code of the new token may fall on either side of a
        # rounding boundary, which moves it by one step of 1/127
        return {"rel": 1e-4, "max": 1e-2, "differ": 1e-3}
    if c["kind"] == "attend":
        return {"rel": 1e-5, "max": 4e-4}    # the appended rows are exact, the softmax sums are fp32
    return {"rel": 1e-5, "max": 4e-4}    # fp32 sums over K
