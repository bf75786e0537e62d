"""What this package's speed is judged by: a dozen programs over its public entry points.

Each case runs one program: a short chain of the callables that `B200Backend` hands to the
evaluation harness and to `BackendBench.enable` (one per aten overload), in the order in
which a model's forward and backward pass, or the evaluation sweep, calls them. `listed()`
names the cases, `draw(rng)` gives further ones of the same programs and ranges, `prepare`
makes the inputs a caller has in hand, `run` is one pass and returns every result in full.

The overloads are separate calls, so each has to read its operands and write its result:
`work` adds that up over the calls of a pass (each operand once, each result once) and
counts the multiply-adds of the contractions.
"""

import functools
import math
from dataclasses import replace

import torch

from backendbench_b200.backends import B200Backend
from backendbench_b200.cases import sweep_cases
from backendbench_b200.eval import compare_enqueue, decode_record, tolerances_for
from backendbench_b200.opregistry import get_operator

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
ITEMSIZE = {"f32": 4, "bf16": 2, "f16": 2}
DEVICE = "cuda"


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest calls: a handful of values through four elementwise operators, as the
        # scalar-sized parts of a model are. Nothing but the cost of a call.
        {"name": "elementwise_small", "path": "elementwise", "dtype": "f32", "rows": 16, "cols": 16, "layout": "contiguous", "other": "full"},
        # Elementwise operators on a transposed view of a large matrix, with a vector
        # broadcast over the rows (a bias after a transpose).
        {"name": "elementwise_transposed", "path": "elementwise", "dtype": "f32", "rows": 39934, "cols": 1024, "layout": "transposed", "other": "row"},
        # A language model's head: log-probabilities of a vocabulary row, the greedy token,
        # and the gradient back to the logits. 50257 is odd: rows start off any vector grid.
        {"name": "vocab_head", "path": "vocab_head", "dtype": "bf16", "rows": 4096, "cols": 50257, "dim": -1},
        # Layer norm of a training step, forward and backward, at a model's hidden width.
        {"name": "layer_norm_train", "path": "layer_norm", "dtype": "bf16", "rows": 8192, "cols": 4096},
        # Causal attention written with bmm / mul / add / softmax, forward and backward.
        {"name": "attention_train", "path": "attention", "dtype": "bf16", "batch": 32, "queries": 2048, "keys": 2048, "head": 128, "train": True},
        # A linear layer's training step at prefill size: output, both gradients, bias gradient.
        {"name": "linear_train", "path": "linear_train", "dtype": "bf16", "rows": 8192, "inner": 4096, "outer": 11008},
        # The same step in fp32 with sizes off every tile and vector grid.
        {"name": "linear_train_f32_ragged", "path": "linear_train", "dtype": "f32", "rows": 1531, "inner": 1027, "outer": 2050},
        # An MLP block while decoding: a few tokens against two large weight matrices.
        {"name": "mlp_decode", "path": "mlp_forward", "dtype": "bf16", "rows": 16, "inner": 4096, "outer": 11008},
        # Token embedding of a training step: table rows out, table gradient back; token ids
        # are as skewed as text is (the most frequent id is about 6 % of all tokens).
        {"name": "embedding_train", "path": "embedding", "dtype": "bf16", "table": 128256, "width": 4096, "tokens": 16384},
        # Element-wise indexing over a square matrix.
        {"name": "indexing_wide", "path": "indexing", "dtype": "f32", "rows": 4096, "cols": 4096, "dim": 0, "picks": 4096},
        # The same on a tall and narrow matrix (features of graph nodes).
        {"name": "indexing_tall", "path": "indexing", "dtype": "f16", "rows": 150134, "cols": 63, "dim": 0, "picks": 75067},
        # The evaluation sweep's many small operator cases, each result compared on the device
        # with its reference: what the harness spends most of its cases on.
        {"name": "sweep_small", "path": "sweep", "sweep_seed": 0, "count": 24, "max_log2": 18},
    ]


PATHS = ("elementwise", "vocab_head", "layer_norm", "attention", "linear_train", "mlp_forward", "embedding", "indexing", "sweep")


def draw(rng):
    """One more case: a program by turns of the die, its sizes spread over their logarithm."""
    budget = 0.6 * _roofline_s(next(c for c in listed() if c["name"] == "linear_train"))
    while True:
        case = _draw_once(rng)
        if _roofline_s(case) <= budget:
            return case


def _draw_once(rng):
    path = rng.choice(PATHS)
    dtype = rng.choice(("bf16", "bf16", "f16", "f32"))
    case = {"path": path, "dtype": dtype}
    if path == "elementwise":
        case.update(rows=_size(rng, 1, 40000), cols=_size(rng, 8, 8192), layout=rng.choice(("contiguous", "contiguous", "transposed")), other=rng.choice(("full", "row", "column")))
    elif path == "vocab_head":
        case.update(rows=_size(rng, 1, 8192), cols=_size(rng, 16, 131072), dim=rng.choice((-1, -1, -1, 0)))
    elif path == "layer_norm":
        case.update(rows=_size(rng, 1, 65536), cols=_size(rng, 16, 8192))
    elif path == "attention":
        queries = _size(rng, 1, 2048)
        case.update(batch=_size(rng, 1, 64), queries=queries, keys=max(queries, _size(rng, 16, 4096)), head=rng.choice((32, 64, 80, 96, 128, 256)), train=rng.random() < 0.5)
    elif path in ("linear_train", "mlp_forward"):
        case.update(rows=_size(rng, 1, 8192), inner=_size(rng, 64, 4096), outer=_size(rng, 64, 11008))
    elif path == "embedding":
        case.update(table=_size(rng, 16, 131072), width=_size(rng, 8, 4096), tokens=_size(rng, 1, 32768))
    elif path == "indexing":
        rows = _size(rng, 8, 160000)
        case.update(rows=rows, cols=_size(rng, 8, 8192), dim=rng.choice((0, 0, 1)), picks=max(1, int(rows * rng.choice((0.5, 1.0)))))
    else:
        case = {"path": path, "sweep_seed": rng.randrange(1, 1 << 20), "count": rng.randint(8, 24), "max_log2": rng.randint(12, 22)}
    return case


def _size(rng, low, high):
    """An extent between `low` and `high`, even in its logarithm; half of them are rounded to
    the multiples of 64 or 8 that models are built with, the others stay as odd as they come."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    grid = rng.choice((64, 8, 1, 1))
    return min(max(n // grid * grid, grid if grid <= n else n, low), high)


def _roofline_s(case):
    w = work(case)
    if case["path"] in ("elementwise", "indexing") and case["rows"] * case["cols"] > 1 << 26:
        return math.inf  # the sweep's largest tensor is 2^26 elements
    if case["path"] == "vocab_head" and case["rows"] * case["cols"] > 1 << 28:
        return math.inf
    if case["path"] == "layer_norm" and case["rows"] * case["cols"] > 1 << 26:
        return math.inf
    return max(w["bytes"] / 6.5e12, w["flops"] / (2.0e14 if case.get("dtype") == "f32" else 1.3e15))


# ------------------------------------------------------------------------------- prepare
@functools.lru_cache(maxsize=None)
def _callables():
    backend = B200Backend()
    names = (
        "relu.default", "add.Tensor", "mul.Tensor", "where.self", "_softmax.default", "_log_softmax.default", "sum.dim_IntList", "native_layer_norm.default",
        "argmax.default", "embedding.default", "index_select.default", "gather.default", "scatter_add.default", "mm.default", "addmm.default", "bmm.default",
        "_softmax_backward_data.default", "_log_softmax_backward_data.default", "native_layer_norm_backward.default", "embedding_dense_backward.default",
    )
    return {n: backend[get_operator(n)] for n in names}


def _sweep_specs(case):
    """The sweep's cases with finite inputs only: a comparison of two results by norms has no
    use for the ones that carry NaN and infinities."""
    specs = sweep_cases(4 * case["count"], case["sweep_seed"], float(case["max_log2"]))
    return [s for s in specs if s.edge != "naninf"][: case["count"]]


def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    dt = DTYPES.get(case.get("dtype"))

    def normal(*shape, std=1.0, mean=0.0):
        return torch.randn(shape, generator=g, device=DEVICE).mul_(std).add_(mean).to(dt)

    def below(high, *shape):
        return torch.randint(0, high, shape, generator=g, device=DEVICE)

    path = case["path"]
    st = {"case": case, "op": _callables()}
    if path == "elementwise":
        r, c = case["rows"], case["cols"]
        st["a"] = normal(c, r).t() if case["layout"] == "transposed" else normal(r, c)
        st["b"] = normal(*{"full": (r, c), "row": (c,), "column": (r, 1)}[case["other"]])
        st["cond"] = torch.rand((r, c), generator=g, device=DEVICE) < 0.5
    elif path == "vocab_head":
        st["logits"] = normal(case["rows"], case["cols"], std=2.0)
        st["grad"] = normal(case["rows"], case["cols"], std=1.0 / case["rows"])
    elif path == "layer_norm":
        r, c = case["rows"], case["cols"]
        st["x"], st["dy"] = normal(r, c), normal(r, c)
        st["w"], st["b"] = normal(c, std=0.02, mean=1.0), normal(c, std=0.02)
    elif path == "attention":
        b, lq, lk, d = case["batch"], case["queries"], case["keys"], case["head"]
        st["q"], st["k"], st["v"] = normal(b, lq, d), normal(b, lk, d), normal(b, lk, d)
        st["scale"] = 1.0 / math.sqrt(d)
        # query i stands at position i + lk - lq and sees the keys up to its own position
        later = torch.arange(lk, device=DEVICE)[None, :] > torch.arange(lq, device=DEVICE)[:, None] + (lk - lq)
        st["mask"] = torch.zeros((1, lq, lk), device=DEVICE).masked_fill_(later[None], -3e4).to(dt)
        if case["train"]:
            st["dout"] = normal(b, lq, d)
    elif path == "linear_train":
        m, k, n = case["rows"], case["inner"], case["outer"]
        st["x"], st["dy"] = normal(m, k), normal(m, n)
        st["w"], st["b"] = normal(n, k, std=1.0 / math.sqrt(k)), normal(n, std=0.02)  # [outer, inner], as torch.nn.Linear keeps it
    elif path == "mlp_forward":
        m, k, n = case["rows"], case["inner"], case["outer"]
        st["x"] = normal(m, k)
        st["w1"], st["b1"] = normal(n, k, std=1.0 / math.sqrt(k)), normal(n, std=0.02)
        st["w2"], st["b2"] = normal(k, n, std=1.0 / math.sqrt(n)), normal(k, std=0.02)
    elif path == "embedding":
        v, d, n = case["table"], case["width"], case["tokens"]
        st["table"], st["grad"] = normal(v, d, std=0.02), normal(n, d)
        # Zipf: the share of id i falls as 1 / (i + 1); frequent ids come first, as in a tokenizer's table
        u = torch.rand((n,), generator=g, device=DEVICE, dtype=torch.float64)
        st["ids"] = torch.exp(u * math.log(v + 1)).long().sub_(1).clamp_(0, v - 1)
    elif path == "indexing":
        r, c, p = case["rows"], case["cols"], case["picks"]
        st["x"], st["src"] = normal(r, c), normal(p, c)
        st["index"] = below((r, c)[case["dim"]], p, c)
        st["picked"] = below(r, p)
    else:
        st["tests"] = []
        for i, spec in enumerate(_sweep_specs(case)):
            spec = replace(spec, seed=seed * 1009 + i)
            args, kwargs = spec.build(DEVICE)
            op = get_operator(spec.op)
            ref = op(*args, **kwargs)
            first = ref[0] if isinstance(ref, tuple) else ref
            st["tests"].append((st["op"][spec.op], args, kwargs, ref, tolerances_for(op, first.dtype)))
        st["records"] = torch.zeros((len(st["tests"]), 8), dtype=torch.int32, device=DEVICE)
    return st


# ----------------------------------------------------------------------------------- run
def run(state):
    return _PROGRAMS[state["case"]["path"]](state, state["op"], state["case"])


def _run_elementwise(st, op, case):
    a, b = st["a"], st["b"]
    total = op["add.Tensor"](a, b, alpha=0.5)
    kept = op["relu.default"](total)
    scaled = op["mul.Tensor"](a, b)
    return total, kept, scaled, op["where.self"](st["cond"], kept, scaled)


def _run_vocab_head(st, op, case):
    dim = case["dim"]
    logp = op["_log_softmax.default"](st["logits"], dim, False)
    token = op["argmax.default"](st["logits"], dim)
    dlogits = op["_log_softmax_backward_data.default"](st["grad"], logp, dim, logp.dtype)
    return logp, token, dlogits


def _run_layer_norm(st, op, case):
    cols = [case["cols"]]
    y, mean, rstd = op["native_layer_norm.default"](st["x"], cols, st["w"], st["b"], 1e-5)
    dx, dw, db = op["native_layer_norm_backward.default"](st["dy"], st["x"], cols, mean, rstd, st["w"], st["b"], [True, True, True])
    return y, mean, rstd, dx, dw, db


def _run_attention(st, op, case):
    bmm, mul = op["bmm.default"], op["mul.Tensor"]
    q, k, v = st["q"], st["k"], st["v"]
    scores = op["add.Tensor"](mul(bmm(q, k.transpose(1, 2)), st["scale"]), st["mask"])
    p = op["_softmax.default"](scores, -1, False)
    out = bmm(p, v)
    if not case["train"]:
        return out
    dout = st["dout"]
    dv = bmm(p.transpose(1, 2), dout)
    dp = bmm(dout, v.transpose(1, 2))
    ds = mul(op["_softmax_backward_data.default"](dp, p, -1, p.dtype), st["scale"])
    return out, bmm(ds, k), bmm(ds.transpose(1, 2), q), dv


def _run_linear_train(st, op, case):
    x, w, dy = st["x"], st["w"], st["dy"]
    y = op["addmm.default"](st["b"], x, w.t())
    dx = op["mm.default"](dy, w)
    dw = op["mm.default"](dy.t(), x)
    return y, dx, dw, op["sum.dim_IntList"](dy, [0])


def _run_mlp_forward(st, op, case):
    hidden = op["relu.default"](op["addmm.default"](st["b1"], st["x"], st["w1"].t()))
    return hidden, op["addmm.default"](st["b2"], hidden, st["w2"].t())


def _run_embedding(st, op, case):
    rows = op["embedding.default"](st["table"], st["ids"])
    return rows, op["embedding_dense_backward.default"](st["grad"], st["ids"], case["table"], -1, False)


def _run_indexing(st, op, case):
    dim, index = case["dim"], st["index"]
    taken = op["gather.default"](st["x"], dim, index)
    summed = op["scatter_add.default"](st["x"], dim, index, st["src"])
    return taken, summed, op["index_select.default"](st["x"], 0, st["picked"])


def _run_sweep(st, op, case):
    results, records = [], st["records"]
    for i, (fn, args, kwargs, ref, (atol, rtol)) in enumerate(st["tests"]):
        res = fn(*args, **kwargs)
        compare_enqueue(ref, res, atol, rtol, records[i])
        results.append(res)
    # the verdicts, read back once for the pass; how far off a last bit is stays out of the outputs
    verdicts = [decode_record(words)[0] == 0 for words in records.tolist()]
    return results, torch.tensor(verdicts)


_PROGRAMS = {
    "elementwise": _run_elementwise,
    "vocab_head": _run_vocab_head,
    "layer_norm": _run_layer_norm,
    "attention": _run_attention,
    "linear_train": _run_linear_train,
    "mlp_forward": _run_mlp_forward,
    "embedding": _run_embedding,
    "indexing": _run_indexing,
    "sweep": _run_sweep,
}


# ------------------------------------------------------------------------ work, tolerance
def work(case):
    es = ITEMSIZE.get(case.get("dtype"), 4)
    path, flops = case["path"], 0
    if path == "elementwise":
        n = case["rows"] * case["cols"]
        nb = {"full": n, "row": case["cols"], "column": case["rows"]}[case["other"]]
        nbytes = es * (2 * (2 * n + nb) + 2 * n + 3 * n) + n  # add, mul; relu; where and its condition
    elif path == "vocab_head":
        n = case["rows"] * case["cols"]
        outs = case["rows"] if case["dim"] == -1 else case["cols"]
        nbytes = es * (2 * n + n + 3 * n) + 8 * outs
    elif path == "layer_norm":
        r, c = case["rows"], case["cols"]
        nbytes = es * (2 * r * c + 2 * c) + 8 * r + es * (3 * r * c + 3 * c) + 8 * r
    elif path == "attention":
        b, lq, lk, d = case["batch"], case["queries"], case["keys"], case["head"]
        s, qd, kd = b * lq * lk, b * lq * d, b * lk * d
        products = 2
        nbytes = es * (qd + kd + s + 2 * s + 2 * s + lq * lk + 2 * s + s + kd + qd)  # q k', scale, mask, softmax, p v
        if case["train"]:
            products = 5
            nbytes += es * ((s + qd + kd) + (qd + kd + s) + 3 * s + 2 * s + (s + kd + qd) + (s + qd + kd))  # dv, dp, ds, scale, dq, dk
        flops = products * 2 * s * d
    elif path == "linear_train":
        m, k, n = case["rows"], case["inner"], case["outer"]
        nbytes = es * (3 * (m * k + k * n + m * n) + n + m * n + n)
        flops = 3 * 2 * m * k * n
    elif path == "mlp_forward":
        m, k, n = case["rows"], case["inner"], case["outer"]
        nbytes = es * (2 * (m * k + k * n + m * n) + n + k + 2 * m * n)
        flops = 2 * 2 * m * k * n
    elif path == "embedding":
        v, d, n = case["table"], case["width"], case["tokens"]
        # a table row that is looked up more than once is read once: as many rows as n ids are expected to hit
        share = torch.log1p(1.0 / torch.arange(1, v + 1, dtype=torch.float64)) / math.log(v + 1)
        hit = int((1.0 - (1.0 - share) ** n).sum())
        nbytes = es * (hit * d + n * d) + 8 * n + es * (n * d + v * d) + 8 * n
    elif path == "indexing":
        r, c, p = case["rows"], case["cols"], case["picks"]
        nbytes = (es * (r * c + p * c) + 8 * p * c) + (es * (2 * r * c + p * c) + 8 * p * c) + (2 * es * p * c + 8 * p)
    else:
        specs = _sweep_specs(case)
        nbytes = flops = 0
        for s in specs:
            nbytes += s.algorithmic_bytes() + 2 * _result_bytes(s)  # the call; both sides of its comparison
            flops += s.flops()
    return {"bytes": nbytes, "flops": flops}


def _result_bytes(spec):
    """Bytes of the result that the comparison reads on each side."""
    es, n = ITEMSIZE[spec.dtype], math.prod(spec.shape)
    op, shape = spec.op, spec.shape
    if op in ("mm.default", "addmm.default"):
        return shape[0] * shape[2] * es
    if op == "bmm.default":
        return shape[0] * shape[1] * shape[3] * es
    if op == "embedding.default":
        return spec.param("n_idx") * shape[1] * es
    if op == "index_select.default":
        return n // max(shape[spec.param("dim", 0)], 1) * spec.param("n_idx") * es
    if op == "gather.default":
        return math.prod(spec.param("index_shape", shape)) * es
    if op == "argmax.default":
        dim = spec.param("dim", -1)
        return 8 * (1 if dim is None else n // max(shape[dim], 1))
    if op == "sum.dim_IntList":
        return n // max(math.prod(shape[d] for d in spec.param("dim")), 1) * es
    return n * es


def tolerance(case):
    path, dtype = case["path"], case.get("dtype")
    if path == "indexing":
        return "exact"  # copies, and sums in the order of the positions that are added
    if path == "sweep":
        return {"rel": 1e-2, "differ": 0.0}  # the coarsest of its data types is bf16
    if path == "embedding":
        return "exact"  # copies, and sums in the order of the tokens
    # about four times the distance from the same programs in 64 bits: one rounding of a 16-bit
    # result is 1.7e-3 (bf16) or 2.2e-4 (f16), a backward attention pass collects 5.6e-3 and 5.9e-4;
    # fp32 products over a few thousand terms come to 2.7e-6
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[dtype]}
