"""Workloads by which the speed of the library is judged.

`listed()` names twelve calls as a program makes them through the public entry points of `cutile_b200`; `draw()` gives
further ones from the same ranges.  Each `kind` below is one path with its own `prepare_*`, `run_*`, `work_*` and
tolerance.  Shapes are in torch order (the Julia shape reversed), inputs have the distributions of the benchmark
configurations, and every array a program would keep between calls (weights, tables, outputs that the entry point takes
as an argument) is made in `prepare`.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("cutile.jl_b200"))  # the package of the tree that is the working folder
import cutile_b200 as ctb  # noqa: E402

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # Prefill of a batch of equal prompts, full multi-head attention: the benchmark's attention configuration.
        dict(name="attention_prefill", kind="attention", dtype="f16", batch=8, heads=16, kv_heads=16, seq_q=1024, seq_kv=1024,
             causal=True),
        # Prefill with grouped key/value heads in bf16; the prompt length is not a multiple of any tile.
        dict(name="attention_prefill_grouped", kind="attention", dtype="bf16", batch=4, heads=32, kv_heads=8, seq_q=2001,
             seq_kv=2001, causal=True),
        # Decode: one new token per sequence against the keys and values of everything before it.
        dict(name="attention_decode", kind="attention", dtype="bf16", batch=32, heads=32, kv_heads=8, seq_q=1, seq_kv=4000,
             causal=True),
        # Expert layer of a serving step with few tokens (router, sort, experts, combine): bound by the expert weights.
        dict(name="moe_256_tokens", kind="moe", tokens=256, hidden=1024, inter=2048, experts=32, topk=2),
        # Expert layer of a prefill or training step: bound by the matrix units.
        dict(name="moe_4096_tokens", kind="moe", tokens=4096, hidden=1024, inter=2048, experts=32, topk=2),
        # Large square product of f32 arrays on TF32 units, the benchmark's dense configuration.
        dict(name="matmul_f32", kind="matmul", dtype="f32", batch=0, m=4096, n=4096, k=4096),
        # Batch of medium products with ragged sizes in bf16: per-head or per-group projections.
        dict(name="batched_matmul_bf16", kind="matmul", dtype="bf16", batch=12, m=1000, n=515, k=776),
        # LayerNorm of a training step, forward and backward with the gradients of weight and bias.
        dict(name="layernorm_train", kind="layernorm", m=4096, n=4096),
        # The smallest call: class probabilities of one small batch, one tile per row.
        dict(name="softmax_classes", kind="softmax", dtype="f32", m=64, n=1000),
        # Probabilities over a vocabulary of odd size: long rows that are not aligned.
        dict(name="softmax_vocabulary", kind="softmax", dtype="f32", m=1024, n=50001),
        # Fused array expression (bias and a tanh-shaped activation) and the column sums its backward pass needs.
        dict(name="tiled_bias_activation", kind="tiled", dtype="f32", rows=8192, cols=4096),
        # Batch of medium transforms, the benchmark's FFT configuration.
        dict(name="fft_batch", kind="fft", batch=256, f0=16, f1=16, f2=16),
    ]


# ------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_attention(rng):
    dtype, heads, group = rng.choice(("f16", "bf16")), rng.choice((8, 16, 32)), rng.choice((1, 4, 8))
    if rng.random() < 0.5:  # decode
        kv = _log(rng, 100, 8192)
        batch = min(_log(rng, 1, 64), max(1, 32 * 8 * 4000 // (heads // group * kv)))
        return dict(kind="attention", dtype=dtype, batch=batch, heads=heads, kv_heads=heads // group, seq_q=1, seq_kv=kv,
                    causal=True)
    causal = rng.random() < 0.75
    seq = _log(rng, 100, 4096 if causal else 2800)
    past = rng.choice((0, 0, _log(rng, 64, 1024)))  # tokens already in the cache: prefill in pieces
    batch = min(_log(rng, 1, 32), max(1, int(4 * 32 * 2001 * 2001 / (heads * seq * (seq + 2 * past) * (1 if causal else 2)))))
    return dict(kind="attention", dtype=dtype, batch=batch, heads=heads, kv_heads=heads // group, seq_q=seq,
                seq_kv=seq + past, causal=causal)


def _draw_moe(rng):
    hidden, inter, experts, topk = rng.choice(((1024, 2048, 32, 2), (512, 1024, 64, 8), (512, 1024, 32, 4), (1024, 2048, 64, 8)))
    return dict(kind="moe", tokens=_log(rng, 1, 8192 // topk), hidden=hidden, inter=inter, experts=experts, topk=topk)


def _draw_matmul(rng):
    dtype = rng.choice(("f32", "f16", "bf16"))
    unit = 16 // BYTES[dtype]  # leading dimensions are multiples of 16 bytes
    m, k = (unit * max(1, _log(rng, 64, 4096) // unit) for _ in range(2))
    n = _log(rng, 64, 4096)
    batch = rng.choice((0, _log(rng, 2, 32)))
    if batch:
        batch = max(1, min(batch, 4096 ** 3 // (m * n * k), 2 ** 26 // (m * k + k * n + m * n)))
    return dict(kind="matmul", dtype=dtype, batch=batch, m=m, n=n, k=k)


def _draw_layernorm(rng):
    n = _log(rng, 256, 8192)
    n = n if rng.random() < 0.25 else n // 4 * 4  # most widths are multiples of four
    return dict(kind="layernorm", m=min(_log(rng, 16, 16384), 4096 * 4096 // n), n=n)


def _draw_softmax(rng):
    dtype, n = rng.choice(("f32", "f32", "f16")), _log(rng, 64, 65536)
    n = n if rng.random() < 0.5 else max(8, n // 8 * 8)
    return dict(kind="softmax", dtype=dtype, m=min(_log(rng, 1, 8192), 1024 * 50001 // n), n=n)


def _draw_tiled(rng):
    cols = _log(rng, 64, 8192)
    cols = cols if rng.random() < 0.25 else cols // 4 * 4
    return dict(kind="tiled", dtype=rng.choice(("f32", "f16")), rows=min(_log(rng, 16, 16384), 8192 * 4096 // cols), cols=cols)


def _draw_fft(rng):
    while True:
        f = [2 ** rng.randint(1, 5) for _ in range(3)]
        n = f[0] * f[1] * f[2]
        if 64 <= n <= 8192:
            return dict(kind="fft", batch=min(_log(rng, 1, 4096), 2 ** 20 // n), f0=f[0], f1=f[1], f2=f[2])


def draw(rng):
    return rng.choice((_draw_attention, _draw_attention, _draw_moe, _draw_matmul, _draw_layernorm, _draw_softmax, _draw_tiled,
                       _draw_fft))(rng)


# ------------------------------------------------------------------ attention
def _prepare_attention(c, g):
    def normal(heads, seq):
        return torch.randn(c["batch"], heads, seq, 64, device="cuda", generator=g).to(DTYPES[c["dtype"]])
    return dict(q=normal(c["heads"], c["seq_q"]), k=normal(c["kv_heads"], c["seq_kv"]), v=normal(c["kv_heads"], c["seq_kv"]),
                options=dict(causal=c["causal"], input_pos=c["seq_kv"] - c["seq_q"] if c["causal"] else 0,
                             query_group_size=c["heads"] // c["kv_heads"]))


def _run_attention(s):
    return ctb.fmha.cutile_fmha(s["q"], s["k"], s["v"], **s["options"])


def _work_attention(c):
    q, kv = c["seq_q"], c["seq_kv"]
    pairs = q * (kv - q) + q * (q + 1) // 2 if c["causal"] else q * kv  # (query, visible key) pairs of a head
    return {"bytes": 2 * 64 * 2 * c["batch"] * (c["heads"] * q + c["kv_heads"] * kv),
            "flops": 4 * 64 * c["batch"] * c["heads"] * pairs}


def _tolerance_attention(c):
    return {"rel": 2e-3 if c["dtype"] == "f16" else 1e-2}


# ------------------------------------------------------------------ mixture of experts
def _prepare_moe(c, g):
    def weight(*shape):
        return torch.randn(*shape, device="cuda", generator=g, dtype=torch.float16).mul_(0.02)
    return dict(x=torch.randn(c["tokens"], c["hidden"], device="cuda", generator=g).half(), topk=c["topk"],
                router=weight(c["experts"], c["hidden"]), w1=weight(c["experts"], 2 * c["inter"], c["hidden"]),
                w2=weight(c["experts"], c["hidden"], c["inter"]))


def _run_moe(s):
    gates, ids = ctb.moe.moe_router(s["x"], s["router"], s["topk"])
    return ctb.moe.cutile_moe(s["x"], s["w1"], s["w2"], gates, ids, 128, 128, 64), gates, ids


def _work_moe(c):
    t, h, i, e, k = (c[n] for n in ("tokens", "hidden", "inter", "experts", "topk"))
    used = e * (1 - (1 - k / e) ** t)  # experts that at least one token picks, for an even router
    return {"bytes": int(2 * (2 * t * h + e * h + used * 3 * h * i)), "flops": 6 * t * k * h * i + 2 * t * h * e}


def _tolerance_moe(c):
    return {"rel": 2e-3}  # the expert ids are whole numbers: they stay the same


# ------------------------------------------------------------------ matrix products
def _prepare_matmul(c, g):
    lead = (c["batch"],) if c["batch"] else ()

    def uniform(*shape):
        return (torch.rand(*lead, *shape, device="cuda", generator=g) * 2 - 1).to(DTYPES[c["dtype"]])
    return dict(a=uniform(c["k"], c["m"]), b=uniform(c["n"], c["k"]), batched=bool(c["batch"]),
                c=torch.empty(*lead, c["n"], c["m"], device="cuda", dtype=DTYPES[c["dtype"]]))


def _run_matmul(s):
    if s["batched"]:
        return ctb.batchmatmul.batch_matmul_kernel(s["a"], s["b"], s["c"], 128, 128, 64)
    return ctb.matmul.matmul_kernel(s["a"], s["b"], s["c"], 64, 64, 64)


def _work_matmul(c):
    m, n, k, batch = c["m"], c["n"], c["k"], c["batch"] or 1
    return {"bytes": BYTES[c["dtype"]] * batch * (m * k + k * n + m * n), "flops": 2 * m * n * k * batch}


def _tolerance_matmul(c):
    return {"rel": {"f32": 2e-3, "f16": 2e-3, "bf16": 1e-2}[c["dtype"]]}  # f32 operands enter with TF32's 10 mantissa bits


# ------------------------------------------------------------------ LayerNorm
def _prepare_layernorm(c, g):
    m, n, groups = c["m"], c["n"], 64

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    def empty(*shape):
        return torch.empty(*shape, device="cuda")
    return dict(x=normal(m, n), dy=normal(m, n), w=torch.rand(n, device="cuda", generator=g) + 0.5, b=normal(n) * 0.1,
                y=empty(m, n), mean=empty(m), rstd=empty(m), dx=empty(m, n), dw_part=empty(groups, n), db_part=empty(groups, n),
                dw=empty(n), db=empty(n), groups=groups)


def _run_layernorm(s):
    ctb.layernorm.layer_norm_fwd(s["x"], s["w"], s["b"], s["y"], s["mean"], s["rstd"], 1e-5, 1024)
    ctb.layernorm.layer_norm_bwd_dx_partial_dwdb(s["dx"], s["dy"], s["dw_part"], s["db_part"], s["x"], s["w"], s["mean"],
                                                 s["rstd"], None, s["groups"], 1024)
    ctb.layernorm.layer_norm_bwd_dwdb(s["dw_part"], s["db_part"], s["dw"], s["db"], 32, 1024)
    return [s[k] for k in ("y", "mean", "rstd", "dx", "dw", "db")]


def _work_layernorm(c):
    m, n = c["m"], c["n"]
    return {"bytes": 4 * (5 * m * n + 5 * n + 4 * m), "flops": 20 * m * n}


def _tolerance_layernorm(c):
    return {"rel": 1e-5}


# ------------------------------------------------------------------ softmax
def _prepare_softmax(c, g):
    x = (torch.randn(c["m"], c["n"], device="cuda", generator=g) * 2).to(DTYPES[c["dtype"]])
    return dict(x=x, out=torch.empty_like(x), n=c["n"], tile=ctb.softmax.next_power_of_2(c["n"]),
                single=c["n"] <= 8192 and c["n"] * BYTES[c["dtype"]] % 16 == 0)


def _run_softmax(s):
    if s["single"]:
        return ctb.softmax.softmax_tma_kernel(s["out"], s["x"], s["tile"])
    return ctb.softmax.softmax_chunked_kernel(s["out"], s["x"], s["n"], 1024)


def _work_softmax(c):
    return {"bytes": 2 * BYTES[c["dtype"]] * c["m"] * c["n"], "flops": 5 * c["m"] * c["n"]}


def _tolerance_softmax(c):
    return {"rel": 1e-5 if c["dtype"] == "f32" else 1e-3}


# ------------------------------------------------------------------ array expressions
def _prepare_tiled(c, g):
    dtype = DTYPES[c["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dtype)
    return dict(x=normal(c["rows"], c["cols"]), bias=normal(c["cols"]), dy=normal(c["rows"], c["cols"]),
                y=torch.empty(c["rows"], c["cols"], device="cuda", dtype=dtype))


def _run_tiled(s):
    T = ctb.tiled
    v = T.Tiled(s["x"]) + T.Tiled(s["bias"])
    T.assign(s["y"], 0.5 * v * (1.0 + T.tanh(0.7978845608 * (v + 0.044715 * (v * v * v)))))
    return s["y"], T.tsum(T.Tiled(s["dy"]), dims=2)


def _work_tiled(c):
    return {"bytes": BYTES[c["dtype"]] * (3 * c["rows"] * c["cols"] + 2 * c["cols"]), "flops": 12 * c["rows"] * c["cols"]}


def _tolerance_tiled(c):
    return {"rel": 1e-5 if c["dtype"] == "f32" else 1e-3}


# ------------------------------------------------------------------ FFT
def _prepare_fft(c, g):
    n = c["f0"] * c["f1"] * c["f2"]
    return dict(x=torch.randn(c["batch"], n, device="cuda", generator=g, dtype=torch.complex64),
                plan=ctb.fft.FftPlan((c["f0"], c["f1"], c["f2"]), "cuda"))


def _run_fft(s):
    return s["plan"](s["x"])


def _work_fft(c):
    n = c["f0"] * c["f1"] * c["f2"]
    return {"bytes": 16 * c["batch"] * n, "flops": int(5 * c["batch"] * n * math.log2(n))}


def _tolerance_fft(c):
    return {"rel": 1e-5}


# ------------------------------------------------------------------ the interface
_RUN = {"attention": _run_attention, "moe": _run_moe, "matmul": _run_matmul, "layernorm": _run_layernorm,
        "softmax": _run_softmax, "tiled": _run_tiled, "fft": _run_fft}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    state = globals()["_prepare_" + case["kind"]](case, g)
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def tolerance(case):
    return globals()["_tolerance_" + case["kind"]](case)
