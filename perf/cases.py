"""The work that users of this package have it do, as cases that can be timed and compared.

Every case goes through a public entry point: a PyTorch function compiled with
``torch.compile`` on this package's Inductor backend (``"kind"`` says which graph), the
tensor-level functions of ``inductor_x_b200.ops``, or the ``b200_graph`` operators.  Sizes are
those of the benchmark configurations and their neighbourhood, odd and ragged ones included.
"""
import math
import types

import torch
import torch.nn.functional as F

import inductor_x_b200  # noqa: F401  (registers the Inductor backend for "cuda")
from inductor_x_b200 import ops
from inductor_x_b200.llama_layer import decoder_layer, rms_norm

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
HEAD = 128  # head dimension of the attention kernels


def listed():
    return [
        # one decoding step's normalisation: a few tokens, so latency is all that counts
        {"name": "rms_norm_decode", "kind": "rms_norm", "dtype": "bf16", "rows": 16, "cols": 4096, "residual": True},
        # benchmark configuration 1: pointwise chain folded into a row sum
        {"name": "gelu_rowsum", "kind": "gelu_rowsum", "dtype": "f32", "rows": 8192, "cols": 1024},
        # benchmark configuration 2, the headline
        {"name": "softmax_layernorm", "kind": "softmax_layernorm", "dtype": "bf16", "rows": 16384, "cols": 4096},
        # the same graph on rows of odd length: no row but the first starts on a 16-byte boundary
        {"name": "softmax_layernorm_ragged", "kind": "softmax_layernorm", "dtype": "f16", "rows": 20011, "cols": 1537},
        # benchmark configuration 3: reductions of a permuted view, and the row gather
        {"name": "permuted_sum", "kind": "permuted_reduce", "op": "sum", "dtype": "f16", "a": 64, "b": 128, "c": 256, "d": 64},
        {"name": "index_select", "kind": "index_select", "dtype": "f16", "rows": 1 << 20, "cols": 128, "picked": 262144},
        # a layout change of the two innermost axes, as between attention layouts
        {"name": "transpose", "kind": "transpose", "dtype": "f16", "a": 4096, "b": 512, "c": 128},
        # normalisation of a training step over 8 x 4096 tokens, forward and backward
        {"name": "rms_norm_training", "kind": "rms_norm_training", "dtype": "bf16", "rows": 32768, "cols": 4096},
        # benchmark configuration 4: causal prefill
        {"name": "attention_prefill", "kind": "attention", "dtype": "bf16", "b": 8, "h": 32, "sq": 4096, "sk": 4096, "causal": True, "layout": "bnsd"},
        # an encoder's attention: no mask, sequence of no whole number of tiles, [B, S, N, D] storage
        {"name": "attention_encoder", "kind": "attention", "dtype": "f16", "b": 16, "h": 16, "sq": 1000, "sk": 1000, "causal": False, "layout": "bsnd"},
        # a training step of configuration 4 on half its batch: output and all three gradients
        {"name": "attention_training", "kind": "attention_training", "dtype": "bf16", "b": 4, "h": 32, "s": 4096, "causal": True},
        # benchmark configuration 5, a whole decoder layer, for one sequence
        {"name": "decoder_layer", "kind": "decoder_layer", "dtype": "bf16", "b": 1, "s": 2048, "heads": 32, "ffn": 11008},
    ]


def _log(rng, low, high):
    """A whole number between low and high, spread over its logarithm, odd ones among them."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["rms_norm", "gelu_rowsum", "softmax_layernorm", "softmax_layernorm", "permuted_reduce", "index_select",
                       "transpose", "rms_norm_training", "attention", "attention", "attention_training", "decoder_layer"])
    half = rng.choice(["f16", "bf16"])
    anyt = rng.choice(["f32", "f16", "bf16"])
    # row lengths are multiples of 64 as often as not: hidden sizes are, vocabularies and sequences are not
    whole = rng.random() < 0.5

    def cols(low, high):
        c = _log(rng, low, high)
        return max(64, c // 64 * 64) if whole else c

    if kind == "rms_norm":
        c = cols(64, 16384)
        return {"kind": kind, "dtype": anyt, "rows": _log(rng, 1, (1 << 26) // c), "cols": c, "residual": rng.random() < 0.5}
    if kind == "gelu_rowsum":
        c = cols(64, 8192)
        return {"kind": kind, "dtype": "f32", "rows": _log(rng, 64, (1 << 25) // c), "cols": c}
    if kind == "softmax_layernorm":
        c = cols(64, 16384)
        return {"kind": kind, "dtype": anyt, "rows": _log(rng, 64, (1 << 26) // c), "cols": c}
    if kind == "permuted_reduce":
        d = rng.choice([16, 32, 64, 64, 96, 128, 256])
        b, c = _log(rng, 16, 512), _log(rng, 16, 512)
        return {"kind": kind, "op": rng.choice(["sum", "amax"]), "dtype": anyt, "a": _log(rng, 1, max(2, (1 << 27) // (b * c * d))), "b": b, "c": c, "d": d}
    if kind == "index_select":
        c = cols(16, 1024)
        return {"kind": kind, "dtype": anyt, "rows": _log(rng, 1024, (1 << 27) // c), "cols": c, "picked": _log(rng, 256, (1 << 26) // c)}
    if kind == "transpose":
        b, c = cols(64, 1024), cols(64, 1024)
        return {"kind": kind, "dtype": anyt, "a": _log(rng, 1, (1 << 27) // (b * c)), "b": b, "c": c}
    if kind == "rms_norm_training":
        c = cols(256, 8192)
        return {"kind": kind, "dtype": half, "rows": _log(rng, 256, (1 << 27) // c), "cols": c}
    if kind == "attention":
        sk = _log(rng, 128, 8192)
        sq = sk if rng.random() < 0.7 else _log(rng, 1, sk)
        heads = max(1, min(256, (1 << 31) // (sq * sk)))
        h = rng.choice([4, 8, 12, 16, 32])
        return {"kind": kind, "dtype": half, "b": _log(rng, 1, max(1, min(32, heads // h))), "h": h, "sq": sq, "sk": sk,
                "causal": rng.random() < 0.6, "layout": rng.choice(["bnsd", "bsnd"])}
    if kind == "attention_training":
        s = _log(rng, 128, 4096)
        h = rng.choice([4, 8, 16, 32])
        return {"kind": kind, "dtype": half, "b": _log(rng, 1, max(1, min(16, (1 << 30) // (s * s * h)))), "h": h, "s": s, "causal": rng.random() < 0.7}
    return {"kind": kind, "dtype": "bf16", "b": rng.choice([1, 2]), "s": _log(rng, 128, 2048), "heads": 32, "ffn": 11008}


# ---- inputs, from the seed alone ----------------------------------------------------------

def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dt, kind = DTYPES[case["dtype"]], case["kind"]

    def normal(*shape, mean=0.0, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * std + mean).to(dt)

    if kind == "rms_norm":
        r, c = case["rows"], case["cols"]
        return [normal(r, c), normal(c, mean=1.0, std=0.1), normal(r, c) if case["residual"] else None]
    if kind == "gelu_rowsum":
        return [normal(case["rows"], case["cols"]), normal(case["cols"]), normal(case["cols"])]
    if kind == "softmax_layernorm":
        c = case["cols"]
        return [normal(case["rows"], c, std=2.0), normal(c, mean=1.0, std=0.1), normal(c, mean=1.0, std=0.1), normal(c, std=0.1)]
    if kind == "permuted_reduce":
        shape = (case["a"], case["b"], case["c"], case["d"])
        return [(torch.rand(*shape, generator=g, device="cuda") * 2 - 1).to(dt)]
    if kind == "index_select":
        table = (torch.rand(case["rows"], case["cols"], generator=g, device="cuda") * 2 - 1).to(dt)
        return [table, torch.randint(0, case["rows"], (case["picked"],), generator=g, device="cuda")]
    if kind == "transpose":
        return [normal(case["a"], case["b"], case["c"])]
    if kind == "rms_norm_training":
        r, c = case["rows"], case["cols"]
        return [normal(r, c), normal(c, mean=1.0, std=0.1), normal(r, c)]
    if kind in ("attention", "attention_training"):
        sq, sk = (case["sq"], case["sk"]) if kind == "attention" else (case["s"], case["s"])

        def heads(s):
            if case.get("layout") == "bsnd":
                return normal(case["b"], s, case["h"], HEAD).transpose(1, 2)
            return normal(case["b"], case["h"], s, HEAD)

        return [heads(sq), heads(sk), heads(sk)] + ([heads(sq)] if kind == "attention_training" else [])
    hidden, ffn = case["heads"] * HEAD, case["ffn"]
    w = {n: normal(hidden, hidden, std=0.02) for n in ("wq", "wk", "wv", "wo")}
    w.update(w_gate=normal(ffn, hidden, std=0.02), w_up=normal(ffn, hidden, std=0.02), w_down=normal(hidden, ffn, std=0.02),
             norm1=normal(hidden, mean=1.0, std=0.1), norm2=normal(hidden, mean=1.0, std=0.1))
    angle = torch.arange(case["s"], device="cuda").float()[:, None] * \
        (1e4 ** (-torch.arange(0, HEAD, 2, device="cuda").float() / HEAD))[None]
    angle = torch.cat([angle, angle], -1)
    return [normal(case["b"], case["s"], hidden), w, angle.cos(), angle.sin()]


# ---- the graphs that are compiled -----------------------------------------------------------

def gelu_rowsum(x, w, b):
    return F.gelu(x * w + b).sum(-1)


def softmax_layernorm(x, g, gamma, beta):
    return F.layer_norm(torch.softmax(x, -1) * g + x, (x.shape[-1],), gamma, beta, 1e-5)


def permuted_sum(x):
    return x.permute(0, 2, 1, 3).sum(3)


def permuted_amax(x):
    return x.permute(0, 2, 1, 3).amax(1)


def index_select(table, idx):
    return table.index_select(0, idx)


def transpose(x):
    return (x.transpose(1, 2) + 1.0).contiguous()


def rms_norm_training(x, w):
    return rms_norm(x, w, 1e-6)


def layer(x, w, cos, sin):
    return decoder_layer(x, w, cos, sin, heads=x.shape[-1] // HEAD)


GRAPHS = {"gelu_rowsum": gelu_rowsum, "softmax_layernorm": softmax_layernorm, "index_select": index_select,
          "transpose": transpose, "rms_norm_training": rms_norm_training, "decoder_layer": layer}
_compiled = {}


def _graph(case):
    """The compiled function of a case, built once per sizes.  Each gets a code object of its own,
    as the graphs of separate programs would have: Dynamo's caches and its limit on
    recompilations go by code object."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    fresh = key not in _compiled
    if fresh:
        fn = (permuted_sum if case["op"] == "sum" else permuted_amax) if case["kind"] == "permuted_reduce" else GRAPHS[case["kind"]]
        own = types.FunctionType(fn.__code__.replace(co_name=f"{fn.__name__}_{len(_compiled)}"), fn.__globals__)
        # (the backend's templates take one order of reduction per kernel; Inductor's fusion of a
        # row sum with the column sum of a weight's gradient is to be left off with this option)
        options = {"triton.mix_order_reduction": False} if case["kind"] == "rms_norm_training" else None
        _compiled[key] = torch.compile(own, dynamic=False, options=options)
    return _compiled[key], fresh


def prepare(case, seed):
    t = _inputs(case, seed)
    kind = case["kind"]
    state = {"case": case, "t": t}
    if kind in ("rms_norm_training", "attention_training"):
        state["wrt"] = t[:2] if kind == "rms_norm_training" else t[:3]
        for x in state["wrt"]:
            x.requires_grad_(True)
    if kind not in ("rms_norm", "attention", "attention_training"):
        state["graph"], fresh = _graph(case)
        if fresh:
            run(state)  # compiles; a user's program has the compiled function in hand
    return state


def run(state):
    case, t = state["case"], state["t"]
    kind = case["kind"]
    if kind == "rms_norm":
        x, w, res = t
        return ops.rmsnorm(x, w, 1e-6, residual=res, return_residual=res is not None)
    if kind == "attention":
        return ops.fused_attention(t[0], t[1], t[2], 1.0 / math.sqrt(HEAD), causal=case["causal"])
    if kind == "attention_training":
        q, k, v, dy = t
        out, _ = torch.ops.b200_graph.b200_sdpa(q, k, v, 1.0 / math.sqrt(HEAD), case["causal"])
        return (out.detach(),) + torch.autograd.grad(out, state["wrt"], dy)
    if kind == "rms_norm_training":
        x, w, dy = t
        out = state["graph"](x, w)
        return (out.detach(),) + torch.autograd.grad(out, state["wrt"], dy)
    return state["graph"](*t)


def work(case):
    kind, e = case["kind"], SIZE[case["dtype"]]
    if kind == "rms_norm":
        n, c = case["rows"] * case["cols"], case["cols"]
        return {"bytes": e * (n * (4 if case["residual"] else 2) + c), "flops": 4 * n}
    if kind == "gelu_rowsum":
        n, c = case["rows"] * case["cols"], case["cols"]
        return {"bytes": e * (n + 2 * c + case["rows"]), "flops": 10 * n}
    if kind == "softmax_layernorm":
        n = case["rows"] * case["cols"]
        return {"bytes": e * (2 * n + 3 * case["cols"]), "flops": 14 * n}
    if kind == "permuted_reduce":
        a, b, c, d = case["a"], case["b"], case["c"], case["d"]
        return {"bytes": e * (a * b * c * d + a * b * (c if case["op"] == "sum" else d)), "flops": a * b * c * d}
    if kind == "index_select":
        distinct = case["rows"] * (1 - math.exp(-case["picked"] / case["rows"]))  # of rows picked at random
        return {"bytes": case["picked"] * 8 + e * case["cols"] * (distinct + case["picked"]), "flops": 0}
    if kind == "transpose":
        return {"bytes": e * 2 * case["a"] * case["b"] * case["c"], "flops": case["a"] * case["b"] * case["c"]}
    if kind == "rms_norm_training":
        n, c = case["rows"] * case["cols"], case["cols"]
        # the forward reads x and writes y, the backward reads x and dy and writes dx; the weight and its gradient
        return {"bytes": e * (5 * n + 3 * c), "flops": 14 * n}
    if kind == "attention":
        sq, sk, heads = case["sq"], case["sk"], case["b"] * case["h"]
        pairs = sq * sk - (sq * (sq - 1) // 2 if case["causal"] else 0)
        return {"bytes": e * HEAD * heads * 2 * (sq + sk), "flops": 4 * HEAD * heads * pairs}
    if kind == "attention_training":
        s, heads = case["s"], case["b"] * case["h"]
        pairs = s * s - (s * (s - 1) // 2 if case["causal"] else 0)
        # q, k, v, out, dout read; out, dq, dk, dv written; two products forward and five backward
        return {"bytes": e * HEAD * heads * s * 9, "flops": 14 * HEAD * heads * pairs}
    tokens, hidden, ffn = case["b"] * case["s"], case["heads"] * HEAD, case["ffn"]
    weights = 4 * hidden * hidden + 3 * hidden * ffn
    pairs = case["b"] * case["heads"] * case["s"] * (case["s"] + 1) // 2
    return {"bytes": e * (weights + 2 * tokens * hidden), "flops": 2 * tokens * weights + 4 * HEAD * pairs}


def tolerance(case):
    kind, dtype = case["kind"], case["dtype"]
    if kind in ("index_select", "transpose") or case.get("op") == "amax":
        return "exact"  # moved values, one rounded addition, or a maximum: nothing depends on an order
    if dtype == "f32":
        return {"rel": 2e-6, "max": 1e-4}
    rounding = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]  # largest relative rounding error of the type
    if kind == "decoder_layer":
        return {"rel": 4 * rounding, "max": 0.1}   # seven products of 16-bit operands in a chain
    if kind in ("attention", "attention_training"):
        return {"rel": 2.5 * rounding, "max": 0.15}   # probabilities and their gradients are 16-bit operands
    return {"rel": 2 * rounding, "max": 6 * rounding}  # 32-bit arithmetic, one rounding of the result


# ---- the same in 64 bits, without this package ------------------------------------------------

def _attention64(q, k, v, causal, dy=None):
    """One (batch, head) at a time: the score matrix of one is all that is held."""
    scale = 1.0 / math.sqrt(HEAD)
    b, h, sq, _ = q.shape
    sk = k.shape[2]
    hidden = torch.ones(sq, sk, dtype=torch.bool, device=q.device).tril(sk - sq).logical_not() if causal else None
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    grads = [torch.empty(t.shape, dtype=torch.float64, device=q.device) for t in (q, k, v)] if dy is not None else []
    for i in range(b):
        for j in range(h):
            qd, kd, vd = (t[i, j].double() for t in (q, k, v))
            p = qd @ kd.T * scale
            if hidden is not None:
                p.masked_fill_(hidden, -math.inf)
            p = torch.softmax(p, -1)
            out[i, j] = p @ vd
            if dy is not None:
                d = dy[i, j].double()
                grads[2][i, j] = p.T @ d
                ds = d @ vd.T
                ds = p * (ds - (ds * p).sum(-1, keepdim=True)) * scale
                grads[0][i, j] = ds @ kd
                grads[1][i, j] = ds.T @ qd
    return (out, *grads) if dy is not None else out


def _by_rows(fn, x, *others):
    """fn over slices of the first axis, so that 64-bit intermediates stay small."""
    step = max(1, (1 << 24) // max(1, x[0].numel()))
    return torch.cat([fn(x[i:i + step].double(), *others) for i in range(0, x.shape[0], step)])


def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w


def exact(case, seed):
    t, kind = _inputs(case, seed), case["kind"]
    if kind == "index_select":
        return t[0].index_select(0, t[1])
    if kind == "transpose":
        # one addition, rounded once: nothing wider to compare it with than the rounded sum itself
        return _by_rows(lambda x: x.transpose(1, 2) + 1.0, t[0])
    if kind == "permuted_reduce":
        return _by_rows(lambda x: x.permute(0, 2, 1, 3).sum(3) if case["op"] == "sum" else x.permute(0, 2, 1, 3).amax(1), t[0])
    if kind == "rms_norm":
        x, w, res = t
        if res is None:
            return _by_rows(lambda x, w: _rms64(x, w), x, w.double())
        # the sum is an output, rounded to the type; the norm is that of the sum in 32 bits or rounded
        h = x.double() + res.double()
        return _rms64(h, w.double()), h
    if kind == "gelu_rowsum":
        return _by_rows(lambda x, w, b: F.gelu(x * w + b).sum(-1), t[0], t[1].double(), t[2].double())
    if kind == "softmax_layernorm":
        def chain(x, g, gamma, beta):
            return F.layer_norm(torch.softmax(x, -1) * g + x, (x.shape[-1],), gamma, beta, 1e-5)
        return _by_rows(chain, t[0], *(p.double() for p in t[1:]))
    if kind == "rms_norm_training":
        x, w, dy = t
        y, dx, dw = [], [], 0
        step = max(1, (1 << 24) // x.shape[1])
        for i in range(0, x.shape[0], step):
            xs, ws = x[i:i + step].double().requires_grad_(True), w.double().requires_grad_(True)
            ys = _rms64(xs, ws)
            gx, gw = torch.autograd.grad(ys, (xs, ws), dy[i:i + step].double())
            y.append(ys.detach())
            dx.append(gx)
            dw = dw + gw
        return torch.cat(y), torch.cat(dx), dw
    if kind == "attention":
        return _attention64(*t, case["causal"])
    if kind == "attention_training":
        return _attention64(t[0], t[1], t[2], case["causal"], t[3])
    x, w, cos, sin = t
    b, s, hidden = x.shape
    x, cos, sin = x.double(), cos.double(), sin.double()

    def heads(y):
        return y.view(b, s, case["heads"], HEAD).transpose(1, 2)

    def rope(y):
        return y * cos + torch.cat([-y[..., HEAD // 2:], y[..., :HEAD // 2]], -1) * sin

    n = _rms64(x, w["norm1"].double())
    q, k, v = (heads(n @ w[name].double().T) for name in ("wq", "wk", "wv"))
    a = _attention64(rope(q), rope(k), v, True).transpose(1, 2).reshape(b, s, hidden)
    hid = x + a @ w["wo"].double().T
    n = _rms64(hid, w["norm2"].double())
    return hid + (F.silu(n @ w["w_gate"].double().T) * (n @ w["w_up"].double().T)) @ w["w_down"].double().T
