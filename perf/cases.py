"""The work this library does for a program that uses it, as cases that can be timed and compared.

Three kinds of callers are covered: a model at inference time (decoder-layer projections at one row, a few rows, a
served batch, a ragged chunk and a whole prefill; the two linears of a Mamba2 block; a whole decode step replayed from a
CUDA graph), the single calls such a model is made of (one small projection, the 4-bit embedding, the online Hadamard
transform) and the load-time work (quantise + pack of a layer, slicing a packed layer to a smaller elastic width).

Weights are N(0, 0.02) quantised round-to-nearest in groups of 128; activations are N(0, 1) with 1 % of the channels
scaled by 20, as the outlier channels of real models are.  Everything is made on the GPU from the case's seed.
"""
import math

import torch
import torch.nn.functional as F

from uniql_b200 import fused, modeling_helpers
from uniql_b200.quantize.quant_embedding_layers import W4O16Embedding
from uniql_b200.quantize.quant_hadamard_layers import Hadamard
from uniql_b200.quantize.quant_linear_layers import W4A16B16O16HadLinear, W4A16B16O16Linear

DEVICE = "cuda"
GROUP = 128

# Layer geometries of the benchmark and the tests: Llama-3.1-8B, the same layer cut to 85 % by structured compression
# (28 of 32 query heads, 12160 of 14336 features: neither is a multiple of 256), Qwen2.5-7B (biases on q/k/v).
LLAMA = dict(hidden=4096, inter=14336, q=4096, kv=1024, bias=False, had=True)
LLAMA85 = dict(hidden=4096, inter=12160, q=3584, kv=1024, bias=False, had=False)
QWEN = dict(hidden=3584, inter=18944, q=3584, kv=512, bias=True, had=False)


def listed():
    return [
        # the smallest call of a decode step: one k or v projection for one token
        dict(name="kv_proj_rows1", op="linear", rows=1, k=4096, n=1024, bias=False, had=False),
        # interactive decoding: the projections of one decoder layer for one token
        dict(name="llama_layer_rows1", op="layer", rows=1, **LLAMA),
        # decoding a small batch, the largest one that still takes the decode kernel
        dict(name="llama_layer_rows16", op="layer", rows=16, **LLAMA),
        # a served batch of decoding requests
        dict(name="llama_layer_rows64", op="layer", rows=64, **LLAMA),
        # a ragged chunk of a prompt on an elastic (compressed) layer
        dict(name="llama85_layer_rows301", op="layer", rows=301, **LLAMA85),
        # a long prompt: the largest case
        dict(name="llama_layer_rows4096", op="layer", rows=4096, **LLAMA),
        # a prompt through the linears of a Mamba2-8B block (8192-point transform in front of out_proj)
        dict(name="mamba2_block_rows2048", op="mamba", rows=2048, hidden=4096, inproj=18560, inner=8192),
        # a whole decode step of Qwen2.5-7B's quantised parts at batch 8: embedding, 28 layers, lm_head, one CUDA graph
        dict(name="qwen_decode_rows8", op="stack", rows=8, layers=28, vocab=152064, **QWEN),
        # the token lookup of a batch of prompts in a 4-bit table
        dict(name="embedding_ids32768", op="embedding", batch=8, seq=4096, vocab=152064, dim=3584),
        # the online transform as a module of its own, over a prompt
        dict(name="hadamard_rows4096", op="hadamard", rows=4096, dim=14336, dtype="float16"),
        # quantising a model layer by layer: one gate projection that already sits on the GPU
        dict(name="quantize_gate", op="quantize", n=14336, k=4096),
        # loading an elastic checkpoint: one decoder layer cut from 32 x 128 / 14336 to 32 x 112 / 12160
        dict(name="slice_llama_layer", op="slice", hidden=4096, heads=32, kv_heads=8, head_dim=128, to_head_dim=112,
             inter=14336, to_inter=12160),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges: row counts over their logarithm, widths that need padding among them."""
    op = rng.choice(["linear", "linear", "linear", "layer", "layer", "layer", "layer", "mamba", "mamba", "stack",
                     "embedding", "hadamard", "hadamard", "quantize", "slice"])
    if op == "linear":
        had = rng.random() < 0.25
        k = rng.choice([2048, 3584, 4096, 5120, 8192, 14336]) if had else _log_int(rng, 256, 14336)
        n = _log_int(rng, 128, 18944)
        rows = _log_int(rng, 1, 4096)
        if rng.random() < 0.5:
            n = max(256, n // 256 * 256)
            k = k if had else max(256, k // 128 * 128)
        return dict(op=op, rows=rows, k=k, n=n, bias=rng.random() < 0.3, had=had)
    if op == "layer":
        geo = dict(rng.choice([LLAMA, LLAMA85, QWEN]))
        if not geo["had"] and rng.random() < 0.5:
            geo["inter"] = rng.randrange(4096, 16384 + 1, 64)
        return dict(op=op, rows=_log_int(rng, 1, 3500), **geo)
    if op == "mamba":
        inner = rng.choice([4096, 8192, 5120])
        return dict(op=op, rows=_log_int(rng, 1, 2048), hidden=4096, inproj=2 * inner + 2 * 8 * 128 + 128, inner=inner)
    if op == "stack":
        return dict(op=op, rows=_log_int(rng, 1, 64), layers=rng.randint(2, 12), vocab=rng.choice([32000, 152064]), **QWEN)
    if op == "embedding":
        return dict(op=op, batch=rng.randint(1, 8), seq=_log_int(rng, 1, 4096), vocab=rng.choice([32000, 128256, 152064]),
                    dim=rng.choice([2048, 3584, 4096, 1000]))
    if op == "hadamard":
        return dict(op=op, rows=_log_int(rng, 1, 4096), dim=rng.choice([1024, 2048, 3584, 4096, 5120, 8192, 14336, 768]),
                    dtype=rng.choice(["float16", "float16", "bfloat16", "float32"]))
    if op == "quantize":
        return dict(op=op, n=_log_int(rng, 512, 18944), k=_log_int(rng, 512, 8192))
    heads, kv_heads = rng.choice([(32, 8), (28, 4)])
    return dict(op=op, hidden=heads * 128, heads=heads, kv_heads=kv_heads, head_dim=128,
                to_head_dim=rng.randrange(64, 128, 8), inter=14336, to_inter=rng.randrange(8192, 14336, 64))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, part):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 1009 + part) % (2 ** 62))


def _weight(seed, part, n, k, std=0.02):
    return (torch.randn(n, k, generator=_gen(seed, part), device=DEVICE) * std).to(torch.float16)


def _bias(seed, part, n):
    return (torch.randn(n, generator=_gen(seed, part), device=DEVICE) * 0.5).to(torch.float16)


def _rows(seed, part, rows, k, dtype=torch.float16):
    g = _gen(seed, part)
    x = torch.randn(rows, k, generator=g, device=DEVICE)
    x *= torch.where(torch.rand(k, generator=g, device=DEVICE) < 0.01, 20.0, 1.0)
    return x.to(dtype)


def _nn_linear(w, b=None):
    lin = torch.nn.Linear(w.shape[1], w.shape[0], bias=b is not None, device="meta")
    lin.weight = torch.nn.Parameter(w, requires_grad=False)
    if b is not None:
        lin.bias = torch.nn.Parameter(b, requires_grad=False)
    return lin


def _layer_parts(case, seed, base=0, out_std=0.02):
    """name -> (weight, bias) of one decoder layer's projections."""
    h, i, q, kv = case["hidden"], case["inter"], case["q"], case["kv"]
    shapes = dict(q=(q, h, 0.02), k=(kv, h, 0.02), v=(kv, h, 0.02), o=(h, q, out_std), gate=(i, h, 0.02), up=(i, h, 0.02),
                  down=(h, i, out_std))
    for j, (name, (n, k, std)) in enumerate(shapes.items()):
        biased = case["bias"] and name in ("q", "k", "v")
        yield name, _weight(seed, base + 2 * j, n, k, std), (_bias(seed, base + 2 * j + 1, n) if biased else None)


def _quantised_layer(case, seed, base=0, out_std=0.02):
    mods = {}
    for name, w, b in _layer_parts(case, seed, base, out_std):
        cls = W4A16B16O16HadLinear if name == "down" and case["had"] else W4A16B16O16Linear
        mods[name] = cls.from_fp16(_nn_linear(w, b))
    return mods


X_PART, TABLE_PART, HEAD_PART, STACK_BASE = 900, 901, 902, 1000


def _stack_std(case):
    # the residual stream stays bounded over the depth when its writers are scaled down with the number of layers
    return 0.02 / math.sqrt(2 * case["layers"])


def prepare(case, seed):
    op = case["op"]
    if op == "linear":
        cls = W4A16B16O16HadLinear if case["had"] else W4A16B16O16Linear
        w, b = _weight(seed, 0, case["n"], case["k"]), _bias(seed, 1, case["n"]) if case["bias"] else None
        return dict(op=op, mod=cls.from_fp16(_nn_linear(w, b)), x=_rows(seed, X_PART, case["rows"], case["k"]))
    if op == "layer":
        return dict(op=op, mods=_quantised_layer(case, seed), x=_rows(seed, X_PART, case["rows"], case["hidden"]))
    if op == "mamba":
        return dict(op=op, in_proj=W4A16B16O16Linear.from_fp16(_nn_linear(_weight(seed, 0, case["inproj"], case["hidden"]))),
                    out_proj=W4A16B16O16HadLinear.from_fp16(_nn_linear(_weight(seed, 1, case["hidden"], case["inner"]))),
                    inner=case["inner"], x=_rows(seed, X_PART, case["rows"], case["hidden"]))
    if op == "stack":
        return _prepare_stack(case, seed)
    if op == "embedding":
        g = _gen(seed, TABLE_PART)
        table = torch.nn.Embedding(case["vocab"], case["dim"], device="meta")
        table.weight = torch.nn.Parameter(_weight(seed, 0, case["vocab"], case["dim"]), requires_grad=False)
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=g, device=DEVICE)
        return dict(op=op, emb=W4O16Embedding.from_fp16(table), ids=ids)
    if op == "hadamard":
        dtype = getattr(torch, case["dtype"])
        return dict(op=op, mod=Hadamard(case["dim"]), x=_rows(seed, X_PART, case["rows"], case["dim"], dtype))
    if op == "quantize":
        return dict(op=op, lin=_nn_linear(_weight(seed, 0, case["n"], case["k"])))
    if op == "slice":
        h, hd = case["hidden"], case["head_dim"]
        geo = dict(hidden=h, inter=case["inter"], q=case["heads"] * hd, kv=case["kv_heads"] * hd, bias=False, had=False)
        return dict(op=op, case=dict(case), mods=_quantised_layer(geo, seed))
    raise ValueError(op)


def _prepare_stack(case, seed):
    table = torch.nn.Embedding(case["vocab"], case["hidden"], device="meta")
    table.weight = torch.nn.Parameter(_weight(seed, TABLE_PART, case["vocab"], case["hidden"], 1.0), requires_grad=False)
    emb = W4O16Embedding.from_fp16(table)
    del table
    layers = [_quantised_layer(case, seed, STACK_BASE + 100 * i, _stack_std(case)) for i in range(case["layers"])]
    head = W4A16B16O16Linear.from_fp16(_nn_linear(_weight(seed, HEAD_PART, case["vocab"], case["hidden"])))
    ids = torch.randint(0, case["vocab"], (case["rows"],), generator=_gen(seed, X_PART), device=DEVICE)

    def step():
        x, kv = emb(ids), []
        for mods in layers:
            _, k, v, _, x = _layer(mods, x, _norm)
            kv.append((k, v))
        return dict(logits=head(_norm(x)), kv=kv)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = step()
    return dict(op="stack", graph=graph, out=out, keep=(emb, layers, head, ids))


# ------------------------------------------------------------------------------------------------ the calls
def _layer(mods, x, norm=None):
    """The projections of one decoder layer (the q rows stand in for the attention result): q, k, v, the residual
    stream after attention and after the MLP.  `norm`: the model's own normalisation, where the layers are chained."""
    norm = norm or (lambda t: t)
    q, k, v = fused.qkv_proj(mods["q"], mods["k"], mods["v"], norm(x))
    y = fused.linear_residual(mods["o"], q, x)
    h = fused.gate_up_swiglu(mods["gate"], mods["up"], norm(y))
    return q, k, v, y, fused.linear_residual(mods["down"], h, y)


def _norm(x):
    return F.rms_norm(x, x.shape[-1:], eps=1e-6)


def run(state):
    op = state["op"]
    if op == "linear":
        return state["mod"](state["x"])
    if op == "layer":
        return _layer(state["mods"], state["x"])
    if op == "mamba":
        zx = state["in_proj"](state["x"])
        return zx, state["out_proj"](zx[:, state["inner"]:2 * state["inner"]])
    if op == "stack":
        state["graph"].replay()
        return state["out"]
    if op == "embedding":
        return state["emb"](state["ids"])
    if op == "hadamard":
        return state["mod"](state["x"])
    if op == "quantize":
        q = W4A16B16O16Linear.from_fp16(state["lin"])
        return q.weight, q.scale
    return _slice(state["case"], state["mods"])


def _slice(c, mods):
    """What the checkpoint loader does to one packed decoder layer, through the slicers it calls."""
    mh, h, hd, to = modeling_helpers, c["hidden"], c["head_dim"], c["to_head_dim"]
    buffers = {n: (m.weight, m.scale, m.workspace) for n, m in mods.items()}
    out = {}
    for n in ("up", "gate"):
        w, s, ws = buffers[n]
        out[n] = mh.slice_w4a16_up_gate_proj(w, s, ws, h, c["inter"], c["to_inter"], w.shape)[:2]
    w, s, ws = buffers["down"]
    out["down"] = mh.slice_w4a16_down_proj(w, s, ws, h, c["inter"], c["to_inter"], w.shape)[:2]
    for n, heads in (("q", c["heads"]), ("k", c["kv_heads"])):
        w, s, ws = buffers[n]
        new_w, _, new_s, _ = mh.slice_w4a16_qk_proj(w, None, s, ws, h, heads, hd, to, w.shape)
        out[n] = (new_w, new_s)
    w, s, ws = buffers["v"]
    out["v"] = mh.slice_w4a16_v_proj(w, s, ws, h, c["kv_heads"], hd, to, w.shape)[:2]
    w, s, ws = buffers["o"]
    out["o"] = mh.slice_w4a16_o_proj(w, s, ws, h, c["heads"], hd, to, w.shape)[:2]
    return out


# ------------------------------------------------------------------------------------------------ what a pass needs
def _linear_work(rows, n, k, had=False):
    """Packed codes + scales read once, rows in and out once; the transform as log2(k) additions per element."""
    nbytes = n * k / 2 + math.ceil(k / GROUP) * n * 2 + rows * (k + n) * 2
    return nbytes, 2.0 * rows * n * k + (rows * k * math.log2(k) if had else 0.0)


def _layer_work(c, rows):
    h, i, q, kv = c["hidden"], c["inter"], c["q"], c["kv"]
    parts = [_linear_work(rows, n, k) for n, k in ((q, h), (kv, h), (kv, h), (h, q), (i, h), (i, h), (h, i))]
    nbytes, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
    # q/k/v and gate/up read the same rows once; the product of gate and up is the only one of the two written;
    # the two residual streams are read once more
    nbytes += rows * 2 * (-3 * h - i + 2 * h)
    return nbytes, flops + (rows * i * math.log2(i) if c["had"] else 0.0)


def work(case):
    op = case["op"]
    if op == "linear":
        nbytes, flops = _linear_work(case["rows"], case["n"], case["k"], case["had"])
    elif op == "layer":
        nbytes, flops = _layer_work(case, case["rows"])
    elif op == "mamba":
        a = _linear_work(case["rows"], case["inproj"], case["hidden"])
        b = _linear_work(case["rows"], case["hidden"], case["inner"], True)
        nbytes, flops = a[0] + b[0], a[1] + b[1]
    elif op == "stack":
        a, b = _layer_work(case, case["rows"]), _linear_work(case["rows"], case["vocab"], case["hidden"])
        nbytes, flops = case["layers"] * a[0] + b[0] + case["rows"] * case["hidden"] * 2.5, case["layers"] * a[1] + b[1]
    elif op == "embedding":
        ids = case["batch"] * case["seq"]
        nbytes, flops = ids * (8 + 2 + case["dim"] * 2.5), ids * case["dim"]
    elif op == "hadamard":
        size = {"float32": 4}.get(case["dtype"], 2)
        nbytes, flops = 2 * size * case["rows"] * case["dim"], case["rows"] * case["dim"] * math.log2(case["dim"])
    elif op == "quantize":
        nk = case["n"] * case["k"]
        nbytes, flops = nk * 2.5 + nk / GROUP * 2, 2.0 * nk
    else:
        h, per = case["hidden"], 0.5 + 2 / GROUP
        kept = (case["heads"] + 2 * case["kv_heads"] + case["heads"]) * case["to_head_dim"] * h + 3 * case["to_inter"] * h
        nbytes, flops = 2 * kept * per, 2.0 * case["heads"] * case["to_head_dim"] * h
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    op = case["op"]
    if op in ("embedding", "quantize", "slice"):
        return "exact"          # one rounding per value, or codes
    if op == "hadamard":
        # one rounding to the output type after 32-bit sums
        return {"float32": {"rel": 1e-6, "max": 1e-5}, "float16": {"rel": 1e-3, "max": 2e-3},
                "bfloat16": {"rel": 8e-3, "max": 2e-2}}[case["dtype"]]
    if op == "linear":
        return {"rel": 1.2e-3, "max": 1e-2}
    if op == "stack":
        # roundings of one layer travel through all that follow
        return {"rel": 1e-2, "max": 8e-2}
    return {"rel": 3e-3, "max": 3e-2}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _dequantised(w):
    """[n, k] fp16 weight -> the group-128 round-to-nearest int4 weight it becomes, (code - 8) * scale in 64 bits.
    The scale is rounded to fp16 where the packed layer stores it and the quotient where the quantiser does."""
    n, k = w.shape
    g = F.pad(w, (0, -k % GROUP)).reshape(n, -1, GROUP)
    scale = g.abs().amax(dim=-1, keepdim=True) * (2 / 15)
    codes = torch.clamp(torch.nan_to_num(torch.round(g / scale), nan=-8.0) + 8, 0, 15) - 8
    return (codes.double() * scale.double()).reshape(n, -1)[:, :k]


def _apply(x, w, b=None):
    """x @ dequantised(w)^T + b in 64 bits, in column slabs that bound the memory."""
    slab = max(256, (1 << 27) // w.shape[1])
    y = torch.cat([x @ _dequantised(w[i:i + slab]).t() for i in range(0, w.shape[0], slab)], dim=1)
    return y if b is None else y + b.double()


def _walsh(x):
    """Natural-order Walsh-Hadamard transform of the last axis (a power of two), unnormalised."""
    n, h = x.shape[-1], 1
    while h < n:
        x = x.reshape(-1, n // (2 * h), 2, h)
        x = torch.stack((x[:, :, 0] + x[:, :, 1], x[:, :, 0] - x[:, :, 1]), dim=2).reshape(-1, n)
        h *= 2
    return x


def _paley(order):
    """The +1/-1 matrix of the orders that are no power of two: Paley I for 12 and 20, Paley II for 28, the Kronecker
    product of the 2-point matrix with the order-20 one for 40."""
    if order == 40:
        h = _paley(20)
        return torch.cat((torch.cat((h, h), 1), torch.cat((h, -h), 1)), 0)
    q = order - 1 if order in (12, 20) else order // 2 - 1
    squares = {a * a % q for a in range(1, q)}
    chi = torch.tensor([[0 if i == j else (1 if (j - i) % q in squares else -1) for j in range(q)] for i in range(q)],
                       dtype=torch.float64)
    one = torch.ones(q, 1, dtype=torch.float64)
    if order in (12, 20):
        s = torch.cat((torch.cat((torch.zeros(1, 1, dtype=torch.float64), one.t()), 1), torch.cat((-one, chi), 1)), 0)
        return s + torch.eye(q + 1, dtype=torch.float64)
    c = torch.cat((torch.cat((torch.zeros(1, 1, dtype=torch.float64), one.t()), 1), torch.cat((one, chi), 1)), 0)
    a, b = torch.tensor([[1.0, 1], [1, -1]], dtype=torch.float64), torch.tensor([[1.0, -1], [-1, -1]], dtype=torch.float64)
    return torch.kron(c, b) + torch.kron(torch.eye(q + 1, dtype=torch.float64), a)


def _hadamard(x):
    """H x / sqrt(dim) in 64 bits, the base matrix on the slow index."""
    dim = x.shape[-1]
    x = x.double()
    if dim & (dim - 1):
        base = next(b for b in (40, 28, 20, 12) if dim % b == 0 and (dim // b) & (dim // b - 1) == 0)
        x = (_paley(base).to(x.device) @ x.reshape(x.shape[0], base, -1)).reshape(x.shape[0] * base, dim // base)
        return _walsh(x).reshape(-1, dim) / math.sqrt(dim)
    return _walsh(x) / math.sqrt(dim)


def _exact_layer(parts, had, x, norm=None):
    norm = norm or (lambda t: t)
    p = {name: (w, b) for name, w, b in parts}
    q, k, v = (_apply(norm(x), *p[n]) for n in ("q", "k", "v"))
    y = x + _apply(q, *p["o"])
    h = F.silu(_apply(norm(y), *p["gate"])) * _apply(norm(y), *p["up"])
    if had:
        h = _hadamard(h)
    return q, k, v, y, y + _apply(h, *p["down"])


def exact(case, seed):
    op = case["op"]
    if op == "linear":
        x = _rows(seed, X_PART, case["rows"], case["k"]).double()
        x = _hadamard(x) if case["had"] else x
        return _apply(x, _weight(seed, 0, case["n"], case["k"]), _bias(seed, 1, case["n"]) if case["bias"] else None)
    if op == "layer":
        return _exact_layer(_layer_parts(case, seed), case["had"], _rows(seed, X_PART, case["rows"], case["hidden"]).double())
    if op == "mamba":
        zx = _apply(_rows(seed, X_PART, case["rows"], case["hidden"]).double(), _weight(seed, 0, case["inproj"], case["hidden"]))
        h = _hadamard(zx[:, case["inner"]:2 * case["inner"]])
        return zx, _apply(h, _weight(seed, 1, case["hidden"], case["inner"]))
    if op == "stack":
        ids = torch.randint(0, case["vocab"], (case["rows"],), generator=_gen(seed, X_PART), device=DEVICE)
        x, kv = _embedded(_weight(seed, TABLE_PART, case["vocab"], case["hidden"], 1.0)[ids]), []
        for i in range(case["layers"]):
            parts = _layer_parts(case, seed, STACK_BASE + 100 * i, _stack_std(case))
            _, k, v, _, x = _exact_layer(parts, case["had"], x, _norm)
            kv.append((k, v))
        return dict(logits=_apply(_norm(x), _weight(seed, HEAD_PART, case["vocab"], case["hidden"])), kv=kv)
    if op == "embedding":
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=_gen(seed, TABLE_PART), device=DEVICE)
        return _embedded(_weight(seed, 0, case["vocab"], case["dim"])[ids])
    if op == "hadamard":
        return _hadamard(_rows(seed, X_PART, case["rows"], case["dim"], getattr(torch, case["dtype"])))
    return None                 # packed codes, and scales that come with them


def _embedded(w):
    """Rows of the 4-bit table: scale amax / 8 per row (stored in fp16), codes rounded to nearest."""
    scale = w.abs().amax(dim=-1, keepdim=True) / 8
    codes = torch.clamp(torch.round(w / scale + 8), 0, 15) - 8
    return codes.double() * scale.double()
