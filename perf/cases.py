"""What the operators of this package are timed on: the calls a recommendation model makes, from a handful of short
histories to a full training batch.

Five kinds of case, each a pass through the public entry points:

  forward   `hstu_jagged` on packed sequences, inference
  train     `hstu_jagged` and its gradients through autograd: one attention layer's part of a training step
  paged     `hstu_paged`: ranking against histories kept in a paged key/value cache
  dense     `hstu_dense`: the [batch, sequence, head, dim] layout
  linear    `distance_in_linear_silu` and its gradients: the projection in front of the attention
  ln_mul    `ln_mul`: the normalisation and gate behind it

A case is a dict of plain values.  Its sequence lengths come from the case alone (so that its work is known); the seed
decides which user has which length, and every value.
"""
import math

import numpy as np
import torch

import ops_rec_b200 as ops_rec

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}


def _attention(kind, name=None, dtype="bf16", batch=32, heads=4, kv_heads=None, dim_qk=128, dim_v=128, lengths="uniform",
               lo=256, hi=1024, mu=0.0, sigma=0.0, targets=0, rab="none", mask="tril", alpha="1/d", lengths_seed=0,
               **more):
    case = dict(kind=kind, dtype=dtype, batch=batch, heads=heads, kv_heads=kv_heads or heads, dim_qk=dim_qk, dim_v=dim_v,
                lengths=lengths, lo=lo, hi=hi, mu=mu, sigma=sigma, targets=targets, rab=rab, mask=mask, alpha=alpha,
                lengths_seed=lengths_seed, **more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest batch, the fp32 case the operator is checked on: 4 short histories, 2 heads of width 32.  What a
        # developer runs in a notebook; launches and host time are all of it.
        _attention("forward", "forward_golden_fp32", "fp32", 4, 2, dim_qk=32, dim_v=32, lo=1, hi=128),
        # One small online ranking request: 8 users of at most 200 events with their candidates, latency is what counts.
        _attention("forward", "forward_request", batch=8, heads=4, dim_qk=64, dim_v=64, lo=20, hi=200, targets=16),
        # An ordinary inference batch: 32 histories of 256 to 1024 events, 4 heads of 128.
        _attention("forward", "forward_mid"),
        # A large ranking batch: 4096 users, mostly short, with up to 64 candidates each and one position bias for all.
        _attention("forward", "forward_serving", batch=4096, dim_qk=64, dim_v=64, lengths="lognormal", lo=8, hi=2048,
                   mu=math.log(200), sigma=0.8, targets=64, rab="shared"),
        # Long histories, the largest inference batch: 256 users of up to 8192 events, 8 heads.
        _attention("forward", "forward_long", batch=256, heads=8, lengths="lognormal", lo=64, hi=8192,
                   mu=math.log(2048), sigma=0.6),
        # A training step with a learned bias per sequence and candidates: gradients of q, k, v and of the bias.
        _attention("train", "train_rab", targets=32, rab="batch"),
        # A training step on long histories, the largest case of all.
        _attention("train", "train_long", batch=64, heads=8, lengths="lognormal", lo=64, hi=8192, mu=math.log(2048),
                   sigma=0.6, lengths_seed=1),
        # A model whose attention width and value width differ (attention_dim 64, linear_dim 128), in half precision.
        _attention("train", "train_mixed_dims", "fp16", batch=24, dim_qk=64, dim_v=128, lo=100, hi=600),
        # A training step in fp32, as in a numerics study of a small model.
        _attention("train", "train_fp32", "fp32", batch=16, heads=2, dim_qk=64, dim_v=64, lo=50, hi=500),
        # Serving from a paged cache: 4096 users, pages of 128 rows, 16 new events and up to 64 candidates as queries.
        _attention("paged", "paged_serving", batch=4096, dim_qk=64, dim_v=64, lengths="lognormal", lo=8, hi=2048,
                   mu=math.log(200), sigma=0.8, targets=64, page=128, new_rows=16),
        # The input projection of a layer of width 1024 on 65536 tokens, forward and backward.
        dict(name="linear_train", kind="linear", dtype="bf16", rows=65536, width=1024, bias=True),
        # Normalisation and gate on the attention output of 262144 tokens.
        dict(name="ln_mul_large", kind="ln_mul", rows=262144, width=1024),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "train", "train", "train", "paged", "paged", "dense", "linear",
                       "linear", "ln_mul"])
    if kind == "linear":
        width = 16 * _spread(rng, 4, 64)
        return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp16"]), rows=_spread(rng, 200, 65536), width=width,
                    bias=rng.random() < 0.7)
    if kind == "ln_mul":
        width = rng.choice([64, 128, 256, 512, 1000, 1024, 2048])
        return dict(kind=kind, rows=_spread(rng, 256, (1 << 28) // max(width, 1024)), width=width)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    heads = rng.choice([2, 4, 8])
    kv_heads = rng.choice([heads, heads, heads, heads // 2])
    dims = rng.choice([(64, 64), (128, 128), (128, 128), (64, 64), (32, 32), (64, 128), (128, 64)])
    # sequences up to `hi` events, as many as a budget of multiply-adds allows
    hi = _spread(rng, 60, 4000 if dtype != "fp32" else 1000)
    lo = max(1, int(hi * rng.choice([0.05, 0.25, 0.5])))
    square = dims in ((64, 64), (128, 128))
    budget = 6e9 if dtype == "fp32" or not square else (1.2e12 if kind != "train" else 4e11)
    pairs = heads * (sum(dims) * 2) * (lo + hi) ** 2 / 8 * 1.1
    batch = min(_spread(rng, 1, 2048), max(1, int(budget / pairs)))
    rab = rng.choice(["none", "none", "none", "batch"] if kind != "forward" else ["none", "none", "shared", "batch"])
    if rab == "batch" and batch * heads * hi * hi > 1 << 27:
        rab = "none"
    targets = rng.choice([0, 0, _spread(rng, 1, max(1, min(64, lo)))])
    common = dict(dtype=dtype, batch=batch, heads=heads, kv_heads=kv_heads, lo=lo, hi=hi, rab=rab,
                  alpha=rng.choice(["1/d", "1/d", "1/sqrt(d)"]), lengths_seed=rng.randrange(1 << 20))
    if kind == "dense":
        common.update(lengths="equal", lo=hi, kv_heads=heads, alpha="1", mask=rng.choice(["tril", "tril", "custom"]))
        common["batch"] = max(1, batch // 3)
        if common["mask"] == "custom":
            common["rab"] = "none"
            common["batch"] = max(1, min(common["batch"], (1 << 27) // (heads * hi * hi)))
        return _attention(kind, dim_qk=dims[0], dim_v=dims[0], **common)
    if kind == "paged":
        common.update(rab="none", page=rng.choice([32, 128, 128, 256]), new_rows=_spread(rng, 1, 64))
        return _attention(kind, dim_qk=dims[0], dim_v=dims[0], targets=max(1, targets), **common)
    return _attention(kind, dim_qk=dims[0], dim_v=dims[1], targets=targets, **common)


# ------------------------------------------------------------------------------------------------ lengths and work
def _lengths(case):
    """(lengths, targets) of the sequences of a case, in the order they are drawn in."""
    rng = np.random.default_rng(case["lengths_seed"])
    n, lo, hi = case["batch"], case["lo"], case["hi"]
    if case["lengths"] == "lognormal":
        ls = np.clip(np.rint(rng.lognormal(case["mu"], case["sigma"], n)), lo, hi).astype(np.int64)
    elif case["lengths"] == "equal":
        ls = np.full(n, hi, dtype=np.int64)
    else:
        ls = rng.integers(lo, hi + 1, n).astype(np.int64)
    ts = np.minimum(rng.integers(1, case["targets"] + 1, n), ls - 1) if case["targets"] else np.zeros(n, np.int64)
    return ls, np.maximum(ts, 0).astype(np.int64)


def _paged_lengths(case):
    """(cached rows, new history rows among them, targets) of every user of a paged case."""
    ls, ts = _lengths(case)
    cached = np.maximum(ls - ts, 1)
    return cached, np.minimum(cached, case["new_rows"]), ts


def work(case):
    kind = case["kind"]
    if kind == "ln_mul":
        return {"bytes": 12.0 * case["rows"] * case["width"], "flops": 10.0 * case["rows"] * case["width"]}
    if kind == "linear":
        m, k = case["rows"], case["width"]
        n = 4 * k
        # x, weight, bias and the four gradients in; linear_output, the four activations and the gradients out
        return {"bytes": 2.0 * (2 * m * k + 2 * n * k + 3 * m * n) + 8.0 * n * case["bias"], "flops": 6.0 * m * n * k}
    es, hq, hk, dq, dv = (_BYTES[case["dtype"]], case["heads"], case["kv_heads"], case["dim_qk"], case["dim_v"])
    if kind == "paged":
        cached, new, ts = _paged_lengths(case)
        rows, keys = int((new + ts).sum()), int((cached + ts).sum())
        pairs = int((new * (cached - new) + new * (new + 1) // 2 + ts * (cached + 1)).sum())
        return {"bytes": float(es * (rows * hq * (dq + dv) + keys * hk * (dq + dv))), "flops": 2.0 * hq * (dq + dv) * pairs}
    ls, ts = _lengths(case)
    n = ls - ts
    pairs = int((n * (n + 1) // 2 + ts * (n + 1)).sum()) if case["mask"] == "tril" else int((ls * ls).sum())
    tokens, plane = int(ls.sum()), case["hi"] * case["hi"]
    bias = {"none": 0, "batch": hq * pairs, "shared": hq * plane // 2}[case["rab"]]
    if case["mask"] == "custom":
        bias += hq * pairs
    qkv = tokens * (hq * dq + hk * (dq + dv))
    if kind == "train":
        grads = qkv + (hq * plane * case["batch"] if case["rab"] == "batch" else 0)
        return {"bytes": float(es * (qkv + 2 * tokens * hq * dv + bias + grads)),
                "flops": 2.0 * hq * (4 * dq + 3 * dv) * pairs}
    return {"bytes": float(es * (qkv + tokens * hq * dv + bias)), "flops": 2.0 * hq * (dq + dv) * pairs}


# ------------------------------------------------------------------------------------------------ inputs
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    rng = np.random.default_rng(seed)
    dtype = _DTYPES[case.get("dtype", "fp32")]
    kind = case["kind"]

    def rnd(*shape, scale=0.5, grad=False):
        t = torch.empty(*shape, device=dev, dtype=dtype).normal_(0.0, scale, generator=gen)
        return t.requires_grad_(grad)

    def offsets(counts):
        return torch.from_numpy(np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)).to(dev)

    def index(values):
        return torch.from_numpy(np.ascontiguousarray(values, dtype=np.int64)).to(dev)

    if kind == "ln_mul":
        m, k = case["rows"], case["width"]
        return dict(kind=kind, x=rnd(m, k), u=rnd(m, k), gamma=1.0 + rnd(k, scale=0.1), beta=rnd(k, scale=0.1))
    if kind == "linear":
        m, k = case["rows"], case["width"]
        n = 4 * k
        bias = torch.empty(n, device=dev).normal_(0.0, 0.1, generator=gen).requires_grad_(True) if case["bias"] else None
        return dict(kind=kind, x=rnd(m, k, grad=True), weight=rnd(n, k, scale=k ** -0.5, grad=True), bias=bias,
                    split=[n // 4] * 4, grads=[rnd(m, n // 4) for _ in range(4)])

    hq, hk, dq, dv = case["heads"], case["kv_heads"], case["dim_qk"], case["dim_v"]
    alpha = {"1/d": 1.0 / dq, "1/sqrt(d)": dq ** -0.5, "1": 1.0}[case["alpha"]]
    order = rng.permutation(case["batch"])
    if kind == "paged":
        cached, new, ts = (a[order] for a in _paged_lengths(case))
        page = case["page"]
        count = (cached + page - 1) // page
        rows = int((new + ts).sum())
        return dict(kind=kind, q=rnd(rows, hq, dq), k=rnd(rows, hk, dq), v=rnd(rows, hk, dv),
                    cache=rnd(int(count.sum()), 2, page, hk, dq), max_q=int((new + ts).max()),
                    max_k=int((cached + ts).max()), seq_offset=offsets(new + ts), seq_offset_k=offsets(cached + ts),
                    seq_offset_t=offsets(ts), page_offsets=offsets(count), page_ids=index(rng.permutation(int(count.sum()))),
                    last_page_len=index(cached - (count - 1) * page), num_target=index(ts), alpha=alpha)

    ls, ts = (a[order] for a in _lengths(case))
    hi, batch = case["hi"], case["batch"]
    grad = kind == "train"
    bias = None
    if case["rab"] == "batch":
        bias = rnd(batch, hq, hi, hi, scale=0.1, grad=grad)
    elif case["rab"] == "shared":
        bias = rnd(hq, hi, hi, scale=0.1)
    if kind == "dense":
        # the dense operator has no alpha argument: such a model scales its queries itself
        mask = None
        if case["mask"] == "custom":
            mask = (torch.rand(batch, hq, hi, hi, device=dev, generator=gen) < 0.7).to(dtype)
        return dict(kind=kind, q=rnd(batch, hi, hq, dq, scale=0.5 / dq), k=rnd(batch, hi, hk, dq), v=rnd(batch, hi, hk, dv),
                    bias=bias, mask=mask, mask_type=3 if mask is not None else 0, max_seq_len=hi)
    tokens = int(ls.sum())
    state = dict(kind=kind, q=rnd(tokens, hq, dq, grad=grad), k=rnd(tokens, hk, dq, grad=grad),
                 v=rnd(tokens, hk, dv, grad=grad), bias=bias, max_seq_len=hi, seq_offset=offsets(ls), num_context=None,
                 num_target=index(ts) if case["targets"] else None, group=1 if case["targets"] else 0, alpha=alpha)
    if grad:
        state["grad_out"] = rnd(tokens, hq, dv)
        if case["targets"]:   # the backward takes num_context and num_target together
            state["num_context"] = torch.zeros(batch, dtype=torch.int64, device=dev)
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    s = state
    kind = s["kind"]
    attention, activation = ops_rec.ascendc.attention, ops_rec.ascendc.activation
    if kind == "ln_mul":
        return activation.ln_mul(s["x"], s["u"], s["gamma"], s["beta"])
    if kind == "linear":
        outs = activation.distance_in_linear_silu(s["x"], s["weight"], s["bias"], s["split"])
        leaves = [s["x"], s["weight"]] + ([s["bias"]] if s["bias"] is not None else [])
        return list(outs) + list(torch.autograd.grad(outs[:4], leaves, s["grads"]))
    if kind == "paged":
        return attention.hstu_paged(s["q"], s["k"], s["v"], s["cache"], None, None, 0, s["max_q"], s["max_k"], 0.0,
                                    s["seq_offset"], s["seq_offset_k"], s["seq_offset_t"], s["page_offsets"],
                                    s["page_ids"], s["last_page_len"], s["num_target"], 1, s["alpha"])
    if kind == "dense":
        return attention.hstu_dense(s["q"], s["k"], s["v"], s["mask"], s["bias"], s["mask_type"], s["max_seq_len"], 0.0)
    out = attention.hstu_jagged(s["q"], s["k"], s["v"], None, s["bias"], 0, s["max_seq_len"], 0.0, s["seq_offset"],
                                s["num_context"], s["num_target"], s["group"], s["alpha"])
    if kind == "forward":
        return out
    leaves = [s["q"], s["k"], s["v"]] + ([s["bias"]] if s["bias"] is not None else [])
    return [out] + list(torch.autograd.grad(out, leaves, s["grad_out"]))


def tolerance(case):
    # about four times the error against the same pass in 64 bits, over every output of 25 cases of these ranges: at most
    # 2.6e-3 in bf16, 7e-4 in fp16, 6.4e-7 in fp32
    return {"rel": {"bf16": 1e-2, "fp16": 3e-3, "fp32": 3e-6}[case.get("dtype", "fp32")]}
