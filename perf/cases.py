"""Performance cases of the attention path: what an engine asks of pooled_b200 while it serves a model.

A case is one forward pass of a model's attention layers through `AttnEngine`, layer after layer, as an engine's loop
over its layers makes the calls.  The kinds:

  token    one new token of one conversation (`encode_layer` per layer)
  host     the same with host buffers (`encode_step_host`: one upload, all layers, one download)
  batch    one new token of each of several conversations of different lengths (`encode_items` per layer)
  block    a few tokens at once: an accepted token and its drafts, checked together (`encode_layer`, decode mode)
  prompt   a prompt, or the next turn of a conversation, into the cache (`encode_layer`)
  gather   tokens that attend selected cache rows only (`rope_append` + `decode_gather`)

Model shapes are the repository's own: "small" 16 q / 8 kv heads x 128, rotated in full; "moe" 16 / 2 x 256 with 64
rotated dims; "hybrid" 24 / 4 x 256 with 64 rotated dims.  The two last have a sigmoid output gate, which their q
projection delivers interleaved with q, and (norm) a QK head-norm ahead of the rotation.
"""
from __future__ import annotations

import math

import torch

from pooled_b200 import AttnConfig, AttnEngine

SHAPES = {
    "small": dict(nH=16, nKV=8, hd=128, n_rot=128, theta=1e6, gated=False, layers=28),
    "moe": dict(nH=16, nKV=2, hd=256, n_rot=64, theta=1e7, gated=True, layers=10),
    "hybrid": dict(nH=24, nKV=4, hd=256, n_rot=64, theta=1e7, gated=True, layers=16),
}
ACT = {"f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # the first tokens of an answer to a short question, small model: 28 launches with next to nothing to read
        dict(name="token_small_short", kind="token", model="small", ctx=301, cols=1, seqs=1, layers=28, act="f16", kv="f16", norm=False),
        # a token deep in a long conversation, every layer as the model has it: interleaved q and gate, QK head-norm
        dict(name="token_moe_32k", kind="token", model="moe", ctx=32768, cols=1, seqs=1, layers=10, act="f16", kv="f16", norm=True),
        # a host that keeps its activations in host memory and hands the library whole token steps
        dict(name="host_hybrid_4k", kind="host", model="hybrid", ctx=4099, cols=1, seqs=1, layers=16, act="f32", kv="f16", norm=False),
        # int8 caches (engine option kvQ8), chosen to fit longer contexts
        dict(name="token_moe_q8_12k", kind="token", model="moe", ctx=12345, cols=1, seqs=1, layers=10, act="f32", kv="q8", norm=True),
        # f32 caches: what the dense engine keeps for small models
        dict(name="token_small_f32_2k", kind="token", model="small", ctx=2000, cols=1, seqs=1, layers=28, act="f32", kv="f32", norm=False),
        # a server's batch: thirteen conversations of every length, a token for each
        dict(name="batch_moe_13", kind="batch", model="moe", ctx=65536, cols=1, seqs=13, layers=4, act="f16", kv="f16", norm=False),
        # speculative decoding: one accepted token and four drafts against a 16k context
        dict(name="block_hybrid_16k", kind="block", model="hybrid", ctx=16384, cols=5, seqs=1, layers=16, act="f16", kv="f16", norm=False),
        # a long prompt into an empty cache
        dict(name="prompt_hybrid_8k", kind="prompt", model="hybrid", ctx=0, cols=8192, seqs=1, layers=4, act="f16", kv="f16", norm=False),
        # a document of no round length into the small model
        dict(name="prompt_small_3k", kind="prompt", model="small", ctx=0, cols=2999, seqs=1, layers=8, act="f16", kv="f16", norm=False),
        # the next question of a long conversation: a short prompt behind a long context
        dict(name="turn_hybrid_9k", kind="prompt", model="hybrid", ctx=9001, cols=203, seqs=1, layers=8, act="f32", kv="f16", norm=True),
        # a prompt into int8 caches
        dict(name="prompt_hybrid_q8", kind="prompt", model="hybrid", ctx=0, cols=777, seqs=1, layers=2, act="f16", kv="q8", norm=False),
        # sparse attention over selected blocks of a long context, four tokens of one sequence
        dict(name="gather_moe_2k", kind="gather", model="moe", ctx=60000, cols=4, seqs=1, layers=10, act="f32", kv="f16", norm=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "token", "host", "batch", "block", "prompt", "prompt", "gather"])
    model = rng.choice(["small", "moe", "hybrid"])
    c = dict(kind=kind, model=model, ctx=0, cols=1, seqs=1, layers=SHAPES[model]["layers"], act=rng.choice(["f16", "f32"]), kv="f16",
             norm=SHAPES[model]["gated"] and kind != "gather" and rng.random() < 0.5)
    if kind == "token":
        c["kv"] = rng.choice(["f16", "f16", "q8", "f32"] if model == "small" else ["f16", "f16", "q8"])
        c["ctx"] = _log(rng, 60, 16384 if c["kv"] == "f32" else 65536)
    elif kind == "host":
        c["ctx"] = _log(rng, 60, 32768)
    elif kind == "batch":
        c["seqs"] = _log(rng, 2, 24)
        c["ctx"] = _log(rng, 512, 65536 if model == "moe" else 32768)
        c["layers"] = 4
    elif kind == "block":
        c["cols"] = rng.randint(2, 8)
        c["ctx"] = _log(rng, 60, 65536)
    elif kind == "prompt":
        c["layers"] = rng.choice([1, 2, 4])
        c["kv"] = rng.choice(["f16", "f16", "f16", "q8"])
        c["cols"] = _log(rng, 48, 8192) if c["kv"] == "f16" else _log(rng, 48, 1024)
        # half of the prompts open a conversation, half follow an earlier one
        room = 4 * 8192 * 8192 // (2 * c["layers"] * c["cols"]) - c["cols"]      # no costlier than the longest listed prompt
        c["ctx"] = 0 if rng.random() < 0.5 or room < 64 else min(room, _log(rng, 60, 32768 if c["kv"] == "f16" else 4096))
    else:
        c["model"], c["layers"] = "moe", SHAPES["moe"]["layers"]
        c["cols"] = rng.randint(1, 8)
        c["ctx"] = _log(rng, 4096, 65536)
    return c


# ---- sizes ----

def _contexts(case):
    """Cached tokens of each sequence before the pass: of a batch, spread over a factor of 64 below the longest."""
    n, top = case["seqs"], case["ctx"]
    if n == 1:
        return [top]
    # golden-ratio steps: every size of batch holds short, middling and long conversations in no order
    return [top if i == 0 else max(1, int(top * 64.0 ** -math.modf(0.6180339887 * i)[0])) for i in range(n)]


def _picked(case):
    """Rows per column of a gathered pass: some thirty 64-row blocks and the newest rows."""
    return [64 * (31 - c % 3) + c + 1 for c in range(case["cols"])]


def _row_bytes(kv, kv_dim):
    return {"f16": 2 * kv_dim, "q8": kv_dim + kv_dim // 8, "f32": 4 * kv_dim}[kv]


def work(case):
    s, cols = SHAPES[case["model"]], case["cols"] * case["seqs"]
    q_dim, kv_dim, es = s["nH"] * s["hd"], s["nKV"] * s["hd"], 2 if case["act"] == "f16" else 4
    row = 2 * _row_bytes(case["kv"], kv_dim)
    if case["kind"] == "gather":
        rows, seen = sum(_picked(case)), sum(_picked(case))
    else:
        rows = sum(n + case["cols"] for n in _contexts(case))
        seen = sum(n + c + 1 for n in _contexts(case) for c in range(case["cols"]))
    acts = cols * es * (q_dim * (3 if s["gated"] else 2) + 2 * kv_dim)           # q, gate and out; k and v
    return {"bytes": case["layers"] * (rows * row + acts + cols * row), "flops": case["layers"] * 4 * s["nH"] * s["hd"] * seen}


def tolerance(case):
    # about four times what one pass differs from the same pass in float64
    if case["kind"] == "prompt" and case["kv"] == "f16":       # q and the softmax weights are single f16 values
        return {"rel": 1.3e-3, "max": 4e-2}
    if case["act"] == "f16":                                   # the rounding of the outputs
        return {"rel": 8e-4, "max": 2e-3}
    return {"rel": 1e-5, "max": 4e-5}                          # 32-bit sums, q and weights of 22 bits


# ---- state ----

def _fill(eng, case, li, seq, n, g, dev):
    """Rows [0, n) of a sequence: keys with a few outlier channels per head, as real ones have, and normal values."""
    s = SHAPES[case["model"]]
    kv_dim = s["nKV"] * s["hd"]
    for which in ("k", "v"):
        x = torch.empty((n, kv_dim), dtype=torch.float16 if case["kv"] == "f16" else torch.float32, device=dev).normal_(generator=g)
        if which == "k":
            x.view(n, s["nKV"], s["hd"])[:, :, 5::61] *= 3.0
        cache = eng.cache(li, which)[seq, :n]
        if case["kv"] == "f16":
            cache.copy_(x.view(torch.int16))
        elif case["kv"] == "f32":
            cache.copy_(x)
        else:
            b = x.view(n, kv_dim // 32, 32)
            sc = b.abs().amax(2) / 127.0
            cache.copy_((b / sc.unsqueeze(2)).round_().clamp_(-127, 127).view(n, kv_dim).to(torch.int8))
            eng.cache_scales(li, which)[seq, :n].copy_(sc)


def _held(view, eng):
    """A view of a cache does not own it: whoever keeps the view keeps the engine."""
    view.engine = eng
    return view


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    s, layers, ctxs, act = SHAPES[case["model"]], case["layers"], _contexts(case), ACT[case["act"]]
    nH, nKV, hd = s["nH"], s["nKV"], s["hd"]
    cols, q_dim, kv_dim = case["cols"] * case["seqs"], nH * hd, nKV * hd
    eng = AttnEngine(AttnConfig(n_heads=nH, n_kv_heads=nKV, head_dim=hd, n_rot=s["n_rot"], rope_theta=s["theta"], max_seq=max(ctxs) + case["cols"] + 64,
                                n_layers=layers, n_seqs=case["seqs"], act_dtype=act, max_cols=max(8, cols), kv_format=case["kv"]), device=dev.index)
    new = lambda *shape: torch.empty(shape, dtype=torch.float32, device=dev).normal_(generator=g).to(act)
    for li in range(layers):
        for seq, n in enumerate(ctxs):
            if n:
                _fill(eng, case, li, seq, n, g, dev)
        if case["norm"]:
            w = [1.0 + 0.1 * torch.empty(hd, dtype=torch.float32, device=dev).normal_(generator=g) for _ in range(2)]
            eng.set_head_norm(li, w[0], w[1])
    st = {"case": case, "eng": eng, "ctxs": ctxs, "hs": 2 * hd if s["gated"] else hd}
    qs = [new(cols, (2 if s["gated"] else 1) * q_dim) for _ in range(layers)]     # gated: [q of a head, gate of a head] per head
    ks, vs = [new(cols, kv_dim) for _ in range(layers)], [new(cols, kv_dim) for _ in range(layers)]
    if case["kind"] == "host":
        pin = lambda ts: torch.stack(ts).cpu().pin_memory()
        st["q"], st["k"], st["v"] = pin(qs), pin(ks), pin(vs)
        st["gate"] = st["q"][:, :, hd:] if s["gated"] else None
        st["out"] = torch.empty((layers, cols, q_dim), dtype=act).pin_memory()
    else:
        st["q"], st["k"], st["v"] = qs, ks, vs
        st["gate"] = [q[:, hd:] if s["gated"] else None for q in qs]
        st["out"] = [torch.empty((cols, q_dim), dtype=act, device=dev) for _ in range(layers)]
    if case["kind"] == "gather":
        picked, stride = _picked(case), 2052
        lists = torch.zeros((layers, cols, stride), dtype=torch.int32, device=dev)
        for li in range(layers):
            for c, n in enumerate(picked):
                tail = c + 1                                     # the newest rows, this column's own among them
                blocks = torch.randperm(case["ctx"] // 64, generator=g, device=dev)[:(n - tail) // 64].sort().values
                rows = (blocks[:, None] * 64 + torch.arange(64, device=dev)).reshape(-1)
                lists[li, c, 0] = n
                lists[li, c, 1:1 + n] = torch.cat([rows, torch.arange(case["ctx"], case["ctx"] + tail, device=dev)])
        st["lists"] = list(lists)
    # what the pass appends, as the caches show it
    st["new"] = []
    for li in range(layers):
        views = [eng.cache(li, w) for w in "kv"] + ([eng.cache_scales(li, w) for w in "kv"] if case["kv"] == "q8" else [])
        st["new"] += [[_held(t[i, n:n + case["cols"]], eng) for i, n in enumerate(ctxs)] for t in views]
    if case["seqs"] == 1:
        st["new"] = [t[0] for t in st["new"]]
    return st


def run(st):
    case, eng, ctxs, hs = st["case"], st["eng"], st["ctxs"], st["hs"]
    q, k, v, gate, out, kind = st["q"], st["k"], st["v"], st["gate"], st["out"], case["kind"]
    if kind == "host":
        eng.encode_step_host(ctxs[0], q, k, v, gate, out, q_head_stride=hs, gate_head_stride=hs)
    elif kind == "batch":
        items = list(enumerate(ctxs))
        for li in range(case["layers"]):
            eng.encode_items(li, items, q[li], k[li], v[li], gate[li], out=out[li], q_head_stride=hs, gate_head_stride=hs)
    elif kind == "gather":
        for li in range(case["layers"]):
            q_rot = eng.rope_append(li, 0, ctxs[0], q[li], k[li], v[li], q_head_stride=hs)
            eng.decode_gather(li, st["lists"][li], q_rot, gate[li], out=out[li], gate_head_stride=hs)
    else:
        mode = "decode" if kind == "block" else "auto"
        for li in range(case["layers"]):
            eng.encode_layer(li, ctxs[0], q[li], k[li], v[li], gate[li], out=out[li], mode=mode, q_head_stride=hs, gate_head_stride=hs)
    if case["seqs"] == 1 and case["layers"] <= 12:
        return out, st["new"]
    # many layers or sequences: what the first and the last cache took, so that the outputs stay few
    return out, st["new"][0], st["new"][-1]
