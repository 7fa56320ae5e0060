"""What is measured: the work that a user of the package has it do, each through the package's public entry points.

A case is a dict of plain values.  `kind` names the path:

  layer        the four projections of transformer layers stored as trees (fused q/k/v, o, fused gate/up, down), each
               called as a module on activations of `rows` tokens; `graph` replays them from a CUDA graph, as a decode
               loop does, otherwise they are called one by one, as a prefill does
  projections  q, k and v kept as separate trees (a checkpoint that is not fused), called eagerly on one batch
  attention    one decode step's attention over compressed pages, `layers` layers in a CUDA graph, ragged lengths
  pages        a prompt's keys and values written into compressed pages and read back as dense BF16
  experts      a routed expert block (top-k of E experts, SwiGLU)
  convert      a BF16 matrix turned into a tree (checked, as by default) and decoded again
  decode       whole decode steps of a small model, prompt fed token by token; returns the logits

Model dimensions are those the repository benchmarks (hidden 4096 / 32 heads / 8 KV heads / intermediate 12288, and 128
experts top-8 of 2048 x 768); drawn cases take other sizes of the same families.
"""
import math
import os
import sys

import torch
import torch.nn as nn

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "statetree-representation_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import statetree_b200 as statetree                                                       # noqa: E402
from statetree_b200.decoder import DecoderConfig, TreeDecoder                            # noqa: E402
from statetree_b200.experts import TreeExperts                                           # noqa: E402
from statetree_b200.kvcache import PAGE, PageStore, decode_splits                        # noqa: E402
from statetree_b200.linear import TreeLinear, forward_list                               # noqa: E402

DEV = "cuda"
D = 128                                  # head dimension
REC = 1552                               # bytes of a weight record (16 x 64 weights)
PAGE_BYTES = 6400                        # bytes of a 16-token page of one KV head (keys and values)


def listed():
    return [
        # token generation for one user: every projection of a few layers at one activation row, replayed from a graph
        dict(name="layer_b1", kind="layer", layers=4, hidden=4096, heads=32, kv_heads=8, inter=12288, rows=1, graph=True),
        # generation for a batch of users (continuous batching)
        dict(name="layer_b64", kind="layer", layers=4, hidden=4096, heads=32, kv_heads=8, inter=12288, rows=64, graph=True),
        # a chunk of a prompt, or a large decode batch: a row count that no tile divides
        dict(name="layer_b300", kind="layer", layers=4, hidden=4096, heads=32, kv_heads=8, inter=12288, rows=300, graph=False),
        # prefill of a long prompt
        dict(name="layer_b2000", kind="layer", layers=2, hidden=4096, heads=32, kv_heads=8, inter=12288, rows=2000, graph=False),
        # the smallest call: q, k, v of a small unfused model for three rows (a few speculative tokens), called eagerly
        dict(name="projections_b3", kind="projections", hidden=2048, heads=32, kv_heads=4, rows=3),
        # one user with a long conversation: latency of the attention of a decode step
        dict(name="attention_b1_16k", kind="attention", layers=4, seqs=1, ctx=16384, heads=32, kv_heads=8),
        # many users with contexts of different lengths
        dict(name="attention_b32_4k", kind="attention", layers=1, seqs=32, ctx=4096, heads=32, kv_heads=8),
        # a prompt's keys and values into the cache, and the pages back as dense tensors for the prefill attention
        dict(name="pages_8k", kind="pages", tokens=8192, kv_heads=8),
        # routed experts while generating for one user
        dict(name="experts_t1", kind="experts", tokens=1, experts=128, top_k=8, hidden=2048, inter=768, graph=True),
        # routed experts in the prefill of a prompt
        dict(name="experts_t1000", kind="experts", tokens=1000, experts=128, top_k=8, hidden=2048, inter=768, graph=False),
        # conversion of a checkpoint's matrix
        dict(name="convert_4096x12288", kind="convert", rows=4096, cols=12288),
        # whole decode steps (every kernel of the runner) for four users, logits of the last step
        dict(name="decode_b4", kind="decode", layers=4, hidden=4096, heads=32, kv_heads=8, inter=12288, vocab=32768,
             seqs=4, prompt=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng):
    """a dense model's sizes: KV heads divide the heads (at most eight query heads each), intermediate not a power of two"""
    kvh = rng.choice((2, 4, 8))
    return dict(hidden=128 * rng.randint(8, 32), heads=kvh * rng.choice((2, 4)), kv_heads=kvh, inter=64 * rng.randint(32, 192))


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "projections", "attention", "pages", "experts", "convert", "decode"))
    if kind == "layer":
        rows = _log(rng, 1, 2000)
        return dict(kind=kind, layers=2, rows=rows, graph=rows <= 128, **_dims(rng))
    if kind == "projections":
        d = _dims(rng)
        return dict(kind=kind, hidden=d["hidden"], heads=d["heads"], kv_heads=d["kv_heads"], rows=_log(rng, 1, 64))
    if kind == "attention":
        seqs, kvh = _log(rng, 1, 64), rng.choice((2, 4, 8))
        return dict(kind=kind, layers=2, seqs=seqs, ctx=_log(rng, 100, min(16384, 65536 // seqs)), heads=kvh * rng.choice((1, 4, 7, 8)),
                    kv_heads=kvh)
    if kind == "pages":
        return dict(kind=kind, tokens=_log(rng, 16, 8192), kv_heads=rng.choice((2, 4, 8)))
    if kind == "experts":
        tokens = _log(rng, 1, 1000)
        return dict(kind=kind, tokens=tokens, experts=rng.choice((32, 64, 128)), top_k=rng.choice((4, 6, 8)),
                    hidden=128 * rng.randint(8, 16), inter=64 * rng.randint(6, 12), graph=tokens <= 16)
    if kind == "convert":
        return dict(kind=kind, rows=16 * _log(rng, 16, 256), cols=64 * _log(rng, 16, 192))
    return dict(kind=kind, layers=2, vocab=16 * rng.randint(500, 2000), seqs=rng.randint(1, 8), prompt=rng.randint(4, 16), **_dims(rng))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1 + int(seed))


def _weight(gen, rows, cols):
    """N(0, 0.02) with one column in a hundred eight times larger: the spread of exponents that real projections have"""
    w = torch.randn(rows, cols, device=DEV, generator=gen) * 0.02
    big = torch.rand(cols, device=DEV, generator=gen) < 0.01
    return (w * torch.where(big, 8.0, 1.0)).to(torch.bfloat16)


def _acts(gen, rows, cols):
    return torch.randn(rows, cols, device=DEV, generator=gen).to(torch.bfloat16)


def _layer_shapes(c):
    q, kv = c["heads"] * D, c["kv_heads"] * D
    return [(q + 2 * kv, c["hidden"]), (c["hidden"], q), (2 * c["inter"], c["hidden"]), (c["hidden"], c["inter"])]


def _projection_shapes(c):
    q, kv = c["heads"] * D, c["kv_heads"] * D
    return [(q, c["hidden"]), (kv, c["hidden"]), (kv, c["hidden"])]


def _layer_inputs(c, seed):
    gen = _gen(seed)
    W = [_weight(gen, m, n) for _ in range(c["layers"]) for m, n in _layer_shapes(c)]
    return W, [_acts(gen, c["rows"], w.shape[1]) for w in W]


def _projection_inputs(c, seed):
    gen = _gen(seed)
    return [_weight(gen, m, n) for m, n in _projection_shapes(c)], _acts(gen, c["rows"], c["hidden"])


def _kv(gen, tokens, heads):
    """keys with channels of very different size, as after a key norm and rotary embedding; values N(0, 1)"""
    scale = torch.exp(torch.randn(heads, D, device=DEV, generator=gen))
    return ((torch.randn(tokens, heads, D, device=DEV, generator=gen) * scale).to(torch.bfloat16),
            torch.randn(tokens, heads, D, device=DEV, generator=gen).to(torch.bfloat16))


def _attention_inputs(c, seed):
    """per layer (q, K, V of all pages, block table); lengths between half the context and the context"""
    gen = _gen(seed)
    pages = -(-c["ctx"] // PAGE)
    B = c["seqs"]
    lens = torch.randint(max(1, c["ctx"] // 2), c["ctx"] + 1, (B,), device=DEV, generator=gen)
    lens[0] = c["ctx"]
    per = []
    for _ in range(c["layers"]):
        K, V = _kv(gen, B * pages * PAGE, c["kv_heads"])
        q = torch.randn(B, c["heads"], D, device=DEV, generator=gen).to(torch.bfloat16)
        table = torch.randperm(B * pages, device=DEV, generator=gen).to(torch.int32).view(B, pages)
        per.append((q, K, V, table))
    return per, lens.to(torch.int32), pages


def _expert_inputs(c, seed):
    gen = _gen(seed)
    E, H, I, T = c["experts"], c["hidden"], c["inter"], c["tokens"]
    up = torch.stack([_weight(gen, 2 * I, H) for _ in range(E)])
    down = torch.stack([_weight(gen, H, I) for _ in range(E)])
    w, ids = torch.softmax(torch.randn(T, E, device=DEV, generator=gen), -1).topk(c["top_k"], -1)
    return up, down, _acts(gen, T, H), ids, (w / w.sum(-1, keepdim=True)).contiguous()


# ------------------------------------------------------------------------------------------------ prepare / run
def _captured(fn, warm):
    """fn() as a CUDA graph on a side stream, after `warm` eager passes there (what a decode runner does): (graph, outputs)"""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(warm):
            fn()
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = fn()
    return graph, out


def _replayable(state, fn, graph):
    state["fn"] = fn
    if graph:
        state["graph"], state["out"] = _captured(fn, 2)
    return state


def prepare(case, seed):
    c, kind = case, case["kind"]
    state = dict(kind=kind)
    if kind == "layer":
        W, X = _layer_inputs(c, seed)
        mods = nn.ModuleList([TreeLinear.from_weight(w, verify=False) for w in W])
        statetree.prepare(mods, batch_sizes=(c["rows"],))
        return _replayable(state, lambda: [m(x) for m, x in zip(mods, X)], c["graph"])
    if kind == "projections":
        W, x = _projection_inputs(c, seed)
        mods = nn.ModuleList([TreeLinear.from_weight(w, verify=False) for w in W])
        statetree.prepare(mods, batch_sizes=(c["rows"],))
        return _replayable(state, lambda: forward_list(list(mods), x), False)
    if kind == "attention":
        per, lens, pages = _attention_inputs(c, seed)
        B, calls = c["seqs"], []
        splits = decode_splits(B, c["kv_heads"], pages)
        for q, K, V, table in per:
            store = PageStore(B * pages, c["kv_heads"], DEV, pool_blocks=1 << 15)
            store.append(K, V, torch.arange(B * pages * PAGE, device=DEV))
            store.check()
            calls.append((store, q, table))
        scale = 1.0 / math.sqrt(D)
        return _replayable(state, lambda: [s.attention(q, t, lens, scale, splits, None, 4) for s, q, t in calls], True)
    if kind == "pages":
        K, V = _kv(_gen(seed), c["tokens"], c["kv_heads"])
        pages = -(-c["tokens"] // PAGE)
        store = PageStore(pages, c["kv_heads"], DEV, pool_blocks=1 << 15)
        slots = torch.arange(c["tokens"], device=DEV)

        def write_and_read():
            store.append(K, V, slots, True)                  # (pages that are written again keep their escape chains)
            return list(store.dense())
        return _replayable(state, write_and_read, False)
    if kind == "experts":
        up, down, x, ids, w = _expert_inputs(c, seed)
        block = TreeExperts.from_weights(up, down, verify=False)
        block.tables()
        block.tensor_maps()
        return _replayable(state, lambda: block(x, ids, w), c["graph"])
    if kind == "convert":
        W = _weight(_gen(seed), c["rows"], c["cols"])

        def convert():
            t = TreeLinear.from_weight(W)
            return [t.tree, t.dequantize()]
        return _replayable(state, convert, False)
    cfg = DecoderConfig(**{k: c[k] for k in ("layers", "hidden", "heads", "kv_heads", "inter", "vocab")})
    dec = TreeDecoder(cfg, torch.device(DEV, torch.cuda.current_device()), c["seqs"], c["prompt"] + 16, seed=int(seed))
    dec.capture()
    prompt = torch.randint(0, c["vocab"], (c["seqs"], c["prompt"]), device=DEV, generator=_gen(seed))

    def steps():
        dec.reset()
        dec.run(prompt, 0)
        return dec.logits.clone()
    return _replayable(state, steps, False)


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return state["fn"]()


# ------------------------------------------------------------------------------------------------ work / tolerance
def _matrix(m, n, rows):
    """(bytes, flops) of a product with a tree: its records, the activations in, the results out"""
    return (m // 16) * (n // 64) * REC + 2 * rows * (m + n), 2 * rows * m * n


def work(case):
    c, kind = case, case["kind"]
    if kind in ("layer", "projections"):
        shapes = _layer_shapes(c) * c["layers"] if kind == "layer" else _projection_shapes(c)
        both = [_matrix(m, n, c["rows"]) for m, n in shapes]
        return dict(bytes=sum(b for b, _ in both), flops=sum(f for _, f in both))
    if kind == "attention":
        tokens = c["layers"] * c["ctx"] * (1 + 0.75 * (c["seqs"] - 1))      # the first is full, the others 3/4 on average
        return dict(bytes=int(tokens * c["kv_heads"] * PAGE_BYTES / PAGE), flops=int(4 * tokens * c["heads"] * D))
    if kind == "pages":
        n = c["tokens"] * c["kv_heads"]
        return dict(bytes=2 * n * 2 * D * 2 + 2 * n * (PAGE_BYTES // PAGE), flops=0)
    if kind == "experts":
        E, H, I, S = c["experts"], c["hidden"], c["inter"], c["tokens"] * c["top_k"]
        used = E * (1 - (1 - 1 / E) ** S)                                   # experts that some pair goes to
        rec = ((2 * I // 16) * (H // 64) + (H // 16) * (I // 64)) * REC
        return dict(bytes=int(used * rec + 4 * c["tokens"] * H), flops=6 * S * H * I)
    if kind == "convert":
        n = c["rows"] * c["cols"]
        return dict(bytes=2 * (2 * n + n // 1024 * REC), flops=0)
    steps = c["prompt"]
    both = [_matrix(m, n, c["seqs"]) for m, n in _layer_shapes(c) * c["layers"] + [(c["vocab"], c["hidden"])]]
    return dict(bytes=steps * sum(b for b, _ in both), flops=steps * sum(f for _, f in both))


def tolerance(case):
    kind = case["kind"]
    if kind in ("pages", "convert"):
        return "exact"
    if kind in ("layer", "projections"):
        return {"rel": 2e-3}                     # BF16 results of fp32 sums: a rounding step apart here and there
    if kind == "attention":
        return {"rel": 4e-3}                     # the same, behind a softmax
    if kind == "experts":
        return {"rel": 8e-3}                     # two BF16 roundings in between (projections, gate)
    return {"rel": 3e-2}                         # a whole model in BF16: roundings travel through its layers


# ------------------------------------------------------------------------------------------------ 64-bit results
def _product(W, x):
    """x W^T in 64 bits, a slice of W's rows at a time"""
    xd = x.double()
    return torch.cat([xd @ W[i:i + 8192].double().t() for i in range(0, W.shape[0], 8192)], 1)


def _norm(x, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _rope(x, pos, theta=1e6):
    """interleaved pairs (2i, 2i + 1) of x [..., 128] turned by pos * theta^(-2i/128)"""
    ang = pos * theta ** (-torch.arange(0, D, 2, device=DEV, dtype=torch.float64) / D)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1).flatten(-2)


def _decode_exact(c, seed):
    """logits after the last prompt token of the model whose weights TreeDecoder draws from `seed` (all norms one)"""
    gen = torch.Generator(device=DEV)
    count = [0]

    def weight(rows, cols):
        gen.manual_seed(int(seed) * 100003 + count[0])
        count[0] += 1
        return (torch.randn(rows, cols, device=DEV, generator=gen) * 0.02).to(torch.bfloat16)
    B, P, h, q, kv, inter = c["seqs"], c["prompt"], c["hidden"], c["heads"] * D, c["kv_heads"] * D, c["inter"]
    embed = weight(c["vocab"], h)
    prompt = torch.randint(0, c["vocab"], (B, P), device=DEV, generator=_gen(seed))
    x = embed[prompt].double()                                              # [B, P, h]
    causal = torch.ones(P, P, dtype=torch.bool, device=DEV).tril()
    pos = torch.arange(P, device=DEV, dtype=torch.float64)[:, None, None]
    G = c["heads"] // c["kv_heads"]
    lin = lambda W, t: _product(W, t.reshape(B * P, -1)).view(B, P, -1)     # noqa: E731
    for _ in range(c["layers"]):
        n = _norm(x)
        Q, K, V = (lin(weight(m, h), n).view(B, P, -1, D) for m in (q, kv, kv))
        Q, K = _rope(_norm(Q), pos), _rope(_norm(K), pos)
        K, V = (t.repeat_interleave(G, 2) for t in (K, V))
        s = torch.einsum("bihd,bjhd->bhij", Q, K) / math.sqrt(D)
        p = torch.softmax(s.masked_fill(~causal, float("-inf")), -1)
        x = x + lin(weight(h, q), torch.einsum("bhij,bjhd->bihd", p, V).reshape(B, P, q))
        n = _norm(x)
        gate, up = lin(weight(inter, h), n), lin(weight(inter, h), n)
        x = x + lin(weight(h, inter), torch.nn.functional.silu(gate) * up)
    return _product(weight(c["vocab"], h), _norm(x[:, -1]))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "layer":
        W, X = _layer_inputs(c, seed)
        return [_product(w, x) for w, x in zip(W, X)]
    if kind == "projections":
        W, x = _projection_inputs(c, seed)
        return [_product(w, x) for w in W]
    if kind == "attention":
        per, lens, pages = _attention_inputs(c, seed)
        G, out = c["heads"] // c["kv_heads"], []
        for q, K, V, table in per:
            y = torch.empty(q.shape, dtype=torch.float64, device=DEV)
            for b in range(c["seqs"]):
                n = int(lens[b])
                k, v = (t.view(-1, PAGE, c["kv_heads"], D)[table[b].long()].reshape(-1, c["kv_heads"], D)[:n].double() for t in (K, V))
                s = torch.einsum("hgd,nhd->hgn", q[b].double().view(-1, G, D), k) / math.sqrt(D)
                y[b] = torch.einsum("hgn,nhd->hgd", torch.softmax(s, -1), v).reshape(-1, D)
            out.append(y)
        return out
    if kind == "pages":
        K, V = _kv(_gen(seed), c["tokens"], c["kv_heads"])
        pages = -(-c["tokens"] // PAGE)
        full = [torch.zeros(pages * PAGE, c["kv_heads"], D, dtype=torch.float64, device=DEV) for _ in (K, V)]
        for dst, src in zip(full, (K, V)):
            dst[:c["tokens"]] = src.double()
        return [t.view(pages, PAGE, c["kv_heads"], D) for t in full]
    if kind == "experts":
        up, down, x, ids, w = _expert_inputs(c, seed)
        out = torch.zeros(x.shape, dtype=torch.float64, device=DEV)
        for e in range(c["experts"]):
            t, j = (ids == e).nonzero(as_tuple=True)
            if t.numel() == 0:
                continue
            gate, lin = (x[t].double() @ up[e].double().t()).chunk(2, 1)
            y = (torch.nn.functional.silu(gate) * lin) @ down[e].double().t()
            out.index_add_(0, t, y * w[t, j].double()[:, None])
        return out
    if kind == "convert":
        return [None, _weight(_gen(seed), c["rows"], c["cols"]).double()]
    return _decode_exact(c, seed)
