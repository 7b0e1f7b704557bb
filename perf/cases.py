"""Performance cases: the work that a user has this framework do, through its public entry points.

Three levels of use:

* whole models given as exported op graphs (`ModelInstance`, `Decoder`): decode steps of the 16-layer fp32 decoder for one
  request, a few and a full batch, prompts through the same graph, and a single decoder layer;
* one small op graph called with host arrays (`ModelInstance.run`), where latency is all that counts;
* single operators on device tensors (`rmlk_b200.kernels`): MatMul in fp32 and fp16, the elementwise / reduction family and the
  indexing / layout family.

`listed()` has twelve fixed cases, `draw(rng)` gives more of the same ranges, odd sizes among them.
"""
import numpy as np
import torch

from rmlk_b200 import dtypes as dt
from rmlk_b200 import kernels as K
from rmlk_b200 import llama
from rmlk_b200.graphspec import GraphSpec
from rmlk_b200.runtime import ModelInstance

F16, F32, I64 = "f16", "f32", "i64"
TORCH = {F16: torch.float16, F32: torch.float32, I64: torch.int64}
SIZE = {F16: 2, F32: 4, I64: 8}
CFG = llama.LLAMA_1B
LAYER_CFG = llama.LlamaConfig(n_layers=1, vocab=128)  # one layer of the same model; its graph starts behind the embedding


def listed():
    return [
        # one decomposed RMSNorm called with host arrays and answered on the host: the smallest call a user makes
        {"name": "norm-64x2048", "kind": "norm", "rows": 64, "cols": 2048},
        # a single decoder layer, one request: a 128-token prompt, then 32 tokens one by one, each read back
        {"name": "layer-1x128+32", "kind": "layer", "batch": 1, "prompt": 128, "steps": 32},
        # one user at a time: every token's logits come back to the host before the next token is fed
        {"name": "decode-1x512", "kind": "decode", "batch": 1, "context": 512, "steps": 16, "io": "step"},
        # a few users with a ragged context; logits streamed to pinned host memory
        {"name": "decode-7x301", "kind": "decode", "batch": 7, "context": 301, "steps": 16, "io": "stream"},
        # a full serving batch that samples on the device
        {"name": "decode-64x512", "kind": "decode", "batch": 64, "context": 512, "steps": 16, "io": "device"},
        # prompts of a few requests, a ragged length
        {"name": "prefill-3x187", "kind": "prefill", "batch": 3, "tokens": 187},
        # prompts of a larger group: the heaviest call
        {"name": "prefill-16x512", "kind": "prefill", "batch": 16, "tokens": 512},
        # one projection of a small decode batch
        {"name": "matmul-f32-8", "kind": "matmul", "dtype": F32, "m": 8, "k": 2048, "n": 8192},
        # an up projection of an 8B-shaped model over a long prompt
        {"name": "matmul-f32-4096", "kind": "matmul", "dtype": F32, "m": 4096, "k": 4096, "n": 14336},
        # the same operator for a half-precision model's prompt
        {"name": "matmul-f16-512", "kind": "matmul", "dtype": F16, "m": 512, "k": 2048, "n": 8192},
        # every elementwise / reduction operator once over the activations of a 4096-token prompt
        {"name": "pointwise-f32-4096x2048", "kind": "pointwise", "dtype": F32, "rows": 4096, "cols": 2048},
        # every indexing / layout operator once over a large tensor of 64-bit values
        {"name": "layout-i64-64x512x16x64", "kind": "layout", "dtype": I64, "d0": 64, "d1": 512, "d2": 16, "d3": 64},
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = int(round(2.0 ** rng.uniform(np.log2(lo), np.log2(hi))))
    return max(lo, min(hi, v // multiple * multiple)) if multiple > 1 else max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["norm", "layer", "decode", "decode", "prefill", "matmul", "matmul", "pointwise", "layout"])
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 1024), "cols": rng.choice([512, 1000, 2048, 4096])}
    if kind == "layer":
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "prompt": _log_int(rng, 16, 400), "steps": rng.randint(8, 32)}
    if kind == "decode":
        batch = _log_int(rng, 1, 64)
        io = "step" if batch <= 2 else rng.choice(["stream", "device"]) if batch <= 16 else "device"
        return {"kind": kind, "batch": batch, "context": _log_int(rng, 32, 1024), "steps": rng.randint(8, 16), "io": io}
    if kind == "prefill":
        batch = _log_int(rng, 1, 16)
        return {"kind": kind, "batch": batch, "tokens": min(_log_int(rng, 16, 1024), 8192 // batch)}
    if kind == "matmul":
        odd = rng.random() < 0.25  # sizes that are no multiple of anything; the rest as model dimensions are
        return {"kind": kind, "dtype": rng.choice([F32, F16]), "m": _log_int(rng, 1, 4096), "k": _log_int(rng, 256, 8192, 1 if odd else 64),
                "n": _log_int(rng, 256, 14336, 1 if odd else 128)}
    if kind == "pointwise":
        return {"kind": kind, "dtype": rng.choice([F32, F16]), "rows": _log_int(rng, 1, 16384), "cols": rng.choice([64, 520, 1023, 2048, 4096])}
    return {"kind": kind, "dtype": rng.choice([F32, I64]), "d0": _log_int(rng, 1, 64), "d1": _log_int(rng, 8, 600), "d2": _log_int(rng, 2, 32),
            "d3": rng.choice([32, 63, 64, 128])}


# ---------------------------------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------------------------------
class _DeviceArray:
    """A tensor that lives in an instance, as the array interface describes it; keeps the instance alive."""

    def __init__(self, inst, name):
        code, shape, ptr = inst.value_info(name)
        self.inst = inst
        self.__cuda_array_interface__ = {"version": 3, "data": (ptr, False), "shape": tuple(shape), "typestr": dt.to_numpy(code).str, "strides": None}


def _on_device(inst, name):
    return torch.as_tensor(_DeviceArray(inst, name), device="cuda")


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _model(cfg, seed, embedding):
    """Weights on the device and an instance of the decoder's op graph on a stream of its own."""
    weights = llama.make_weights_device(cfg, seed)
    if not embedding:
        weights = {n: w for n, w in weights.items() if n not in ("embed", "lm_head")}
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    dec = llama.Decoder(cfg, llama.build_graph(cfg, weights, device_weights=True, with_embedding=embedding), stream=stream.cuda_stream)
    return {"weights": weights, "stream": stream, "dec": dec}


def _prepare_norm(c, seed):
    rng = np.random.default_rng(seed)
    g = GraphSpec()
    g.input("x", np.float32, [1, 0, c["cols"]])
    g.const("two", np.array(2.0, np.float32))
    g.const("eps", np.array(1e-5, np.float32))
    g.const("weight", (1 + 0.1 * rng.standard_normal(c["cols"])).astype(np.float32))
    g.op("Pow", ["x", "two"], "x2")
    g.op("ReduceMean", ["x2"], "mean", axes=[-1], keepdims=1)
    g.op("Add", ["mean", "eps"], "mean_eps")
    g.op("Sqrt", ["mean_eps"], "deviation")
    g.op("Div", ["x", "deviation"], "unit")
    g.op("Mul", ["unit", "weight"], "y")
    g.output("y")
    return {"inst": ModelInstance(g.to_runtime()), "x": rng.standard_normal((1, c["rows"], c["cols"]), dtype=np.float32)}


def _prepare_layer(c, seed):
    s = _model(LAYER_CFG, seed, embedding=False)
    rng = np.random.default_rng(seed)
    b, p = c["batch"], c["prompt"]
    s["embeds"] = [rng.standard_normal((b, n, LAYER_CFG.hidden), dtype=np.float32) * np.float32(0.02) for n in [p] + [1] * c["steps"]]
    s["masks"] = [np.ones((b, p + i), np.int64) for i in range(c["steps"] + 1)]
    s["positions"] = [np.tile(np.arange(p, dtype=np.int64), (b, 1))] + [np.full((b, 1), p + i, np.int64) for i in range(c["steps"])]
    return s


def _prepare_decode(c, seed):
    """A prompt's KV cache is in hand (kept from an earlier request); the tokens that follow it are given."""
    s = _model(CFG, seed, embedding=True)
    g = _generator(seed + 1)
    b, t, n = c["batch"], c["context"], c["steps"]
    shape = [b, CFG.n_kv_heads, t, CFG.head_dim]
    s["past"] = {f"past_key_values.{l}.{kv}": _randn(g, *shape, scale=0.9) for l in range(CFG.n_layers) for kv in ("key", "value")}
    ids = torch.randint(0, CFG.vocab, (n, b, 1), device="cuda", generator=g)
    if c["io"] == "device":
        s["ids"] = ids
        s["masks"] = [torch.ones(b, t + i + 1, dtype=torch.int64, device="cuda") for i in range(n)]
        s["positions"] = [torch.full((b, 1), t + i, dtype=torch.int64, device="cuda") for i in range(n)]
        s["logits"] = torch.empty(n, b, 1, CFG.vocab, device="cuda")
    else:
        s["ids"] = ids.cpu().numpy()
        if c["io"] == "stream":
            s["logits"] = torch.empty(n, b, 1, CFG.vocab, pin_memory=True)
    return s


def _prepare_prefill(c, seed):
    s = _model(CFG, seed, embedding=True)
    s["ids"] = np.random.default_rng(seed).integers(0, CFG.vocab, (c["batch"], c["tokens"]))
    return s


def _prepare_matmul(c, seed):
    g, m, k, n = _generator(seed), c["m"], c["k"], c["n"]
    d = TORCH[c["dtype"]]
    # fp16 activations at the scale of normalised hidden states, so that products are not subnormal
    a = _randn(g, m, k, scale=0.02 if c["dtype"] == F32 else 1.0, dtype=d)
    b = _randn(g, k, n, scale=0.02, dtype=d)
    bytes_ = K.matmul_workspace_bytes(1, m, n, k) if c["dtype"] == F32 else 0
    return {"a": a, "b": b, "out": torch.empty(m, n, dtype=d, device="cuda"),
            "workspace": torch.empty(bytes_, dtype=torch.uint8, device="cuda") if bytes_ else None}


def _prepare_pointwise(c, seed):
    g, r, n, d = _generator(seed), c["rows"], c["cols"], TORCH[c["dtype"]]
    x, y = _randn(g, r, n, dtype=d), _randn(g, r, n, dtype=d)
    return {"x": x, "y": y, "positive": x.abs() + 0.5, "row": _randn(g, n, dtype=d), "col": _randn(g, r, 1, dtype=d).abs() + 0.5,
            "two": torch.full((), 2.0, dtype=d, device="cuda"), "steps": (x * 2).round(), "steps_y": (y * 2).round(), "flag": x > 0,
            "to": torch.float16 if c["dtype"] == F32 else torch.float32}


def _prepare_layout(c, seed):
    g, d = _generator(seed), TORCH[c["dtype"]]
    shape = [c["d0"], c["d1"], c["d2"], c["d3"]]

    def values(*dims):
        return torch.randint(-(1 << 40), 1 << 40, dims, device="cuda", generator=g) if d == torch.int64 else _randn(g, *dims)

    rows = c["d0"] * c["d1"]
    half = max(1, rows // 2)
    return {"x": values(*shape), "indices": torch.randint(0, rows, (half,), device="cuda", generator=g),
            # each row is written at most once: the result does not depend on the order of the writes
            "places": torch.randperm(rows, device="cuda", generator=g)[:half].reshape(half, 1).contiguous(),
            "updates": values(half, c["d2"] * c["d3"]), "shared": values(c["d0"], 1, c["d2"], c["d3"])}


_PREPARE = {"norm": _prepare_norm, "layer": _prepare_layer, "decode": _prepare_decode, "prefill": _prepare_prefill, "matmul": _prepare_matmul,
            "pointwise": _prepare_pointwise, "layout": _prepare_layout}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["case"] = case
    return state


# ---------------------------------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------------------------------
def _run_norm(c, s):
    return s["inst"].run({"x": s["x"]})


def _run_layer(c, s):
    dec = s["dec"]
    inst = dec.inst
    dec.reset(c["batch"])
    hidden = []
    for x, mask, pos in zip(s["embeds"], s["masks"], s["positions"]):
        inst.set_input("inputs_embeds", x)
        inst.set_input("attention_mask", mask)
        inst.set_input("position_ids", pos)
        inst.launch()
        hidden.append(inst.read("hidden_out"))
    return hidden + [inst.read("present.0.key"), inst.read("present.0.value")]


def _run_decode(c, s):
    dec = s["dec"]
    inst = dec.inst
    b, t = c["batch"], c["context"]
    for name, x in s["past"].items():
        inst.set_input_ptr(name, dt.F32, list(x.shape), x.data_ptr(), True)
    dec.batch, dec.context = b, t
    if c["io"] == "step":
        return [dec.step(ids) for ids in s["ids"]]
    logits = s["logits"]
    if c["io"] == "stream":
        for i, ids in enumerate(s["ids"]):
            inst.stream_output("logits", logits[i].data_ptr(), logits[i].numel() * 4)
            dec.feed(ids)
            inst.launch()
            inst.wait_outputs()
        return logits
    with torch.cuda.stream(s["stream"]):
        for i in range(c["steps"]):
            inst.set_input_ptr("input_ids", dt.I64, [b, 1], s["ids"][i].data_ptr(), True)
            inst.set_input_ptr("attention_mask", dt.I64, [b, t + i + 1], s["masks"][i].data_ptr(), True)
            inst.set_input_ptr("position_ids", dt.I64, [b, 1], s["positions"][i].data_ptr(), True)
            inst.launch()
            logits[i].copy_(_on_device(inst, "logits"))
    return logits


def _run_prefill(c, s):
    dec = s["dec"]
    dec.reset(c["batch"])
    dec.feed(s["ids"])
    dec.inst.launch()
    return _on_device(dec.inst, "logits")


def _run_matmul(c, s):
    return K.matmul(s["a"], s["b"], out=s["out"], workspace=s["workspace"])


def _run_pointwise(c, s):
    x, y, row = s["x"], s["y"], s["row"]
    return [K.binary("add", x, row), K.binary("sub", x, y), K.binary("mul", x, y), K.binary("div", x, s["col"]), K.pow_(x, s["two"]),
            K.binary("equal", s["steps"], s["steps_y"]), K.binary("greater", x, y), K.unary("sqrt", s["positive"]), K.unary("neg", x),
            K.unary("sin", x), K.unary("cos", x), K.unary("sigmoid", x), K.unary("relu", x), K.cast(x, s["to"]), K.where(s["flag"], x, row),
            K.reduce_mean(x, [-1]), K.softmax(x)]


def _run_layout(c, s):
    x = s["x"]
    d0, d1, d2, d3 = x.shape
    flat = x.view(d0 * d1, d2 * d3)
    return [K.gather(flat, s["indices"]), K.scatter_nd(flat, s["places"], s["updates"]),
            K.slice_(x, [d3 // 2], [d3], axes=[3]), K.slice_(x, [1, 0], [d1, d2], axes=[1, 2], steps=[2, 1]),
            K.transpose(x, [0, 2, 1, 3]), K.transpose(x, [0, 1, 3, 2]), K.transpose(x, [3, 2, 1, 0]),
            K.concat([x, s["shared"]], 1), K.expand(s["shared"], [d0, d1, d2, d3])]


_RUN = {"norm": _run_norm, "layer": _run_layer, "decode": _run_decode, "prefill": _run_prefill, "matmul": _run_matmul,
        "pointwise": _run_pointwise, "layout": _run_layout}


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


# ---------------------------------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------------------------------
def _layer_params(cfg):
    q, kv = cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    return 2 * cfg.hidden * q + 2 * cfg.hidden * kv + 3 * cfg.hidden * cfg.ffn


def _pass(cfg, batch, past, new, vocab):
    """Bytes and operations of one pass of `new` tokens per request over `past` cached ones: weights and cache once, the new
    rows and the outputs once; query i of a request sees past + i + 1 keys."""
    per_layer = _layer_params(cfg)
    head = cfg.hidden * vocab
    seen = sum(past + i + 1 for i in range(new))
    kv_row = 2 * cfg.n_kv_heads * cfg.head_dim * 4
    moved = cfg.n_layers * (per_layer * 4 + 2 * cfg.hidden * 4 + batch * kv_row * (past + new)) + head * 4
    moved += batch * new * (2 * cfg.hidden * 4 if not vocab else cfg.hidden * 4 + vocab * 4)
    flops = 2 * batch * new * (cfg.n_layers * per_layer + head) + cfg.n_layers * 4 * batch * cfg.n_heads * cfg.head_dim * seen
    return moved, flops


def work(case):
    c, kind = case, case["kind"]
    if kind == "norm":
        n = c["rows"] * c["cols"]
        return {"bytes": 4 * (2 * n + c["cols"]), "flops": 4 * n}
    if kind == "layer":
        passes = [_pass(LAYER_CFG, c["batch"], 0, c["prompt"], 0)] + [_pass(LAYER_CFG, c["batch"], c["prompt"] + i, 1, 0) for i in range(c["steps"])]
    elif kind == "decode":
        passes = [_pass(CFG, c["batch"], c["context"] + i, 1, CFG.vocab) for i in range(c["steps"])]
    elif kind == "prefill":
        passes = [_pass(CFG, c["batch"], 0, c["tokens"], CFG.vocab)]
    elif kind == "matmul":
        m, k, n = c["m"], c["k"], c["n"]
        return {"bytes": SIZE[c["dtype"]] * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    elif kind == "pointwise":
        n, e = c["rows"] * c["cols"], SIZE[c["dtype"]]
        # full tensors read and written: add, div, pow, softmax 2 each, sub and mul 3, the comparisons 2, six unary operators 2 each, the mean 1
        moved = e * n * (4 * 2 + 2 * 3 + 2 * 2 + 6 * 2 + 1) + 2 * n      # a comparison writes one byte per element
        moved += n * (e + (2 if e == 4 else 4)) + n * (1 + 2 * e) + e * c["rows"]  # cast, where, the means
        return {"bytes": moved, "flops": 17 * n}
    else:
        n, e, row = c["d0"] * c["d1"] * c["d2"] * c["d3"], SIZE[c["dtype"]], c["d2"] * c["d3"]
        half, shared = max(1, c["d0"] * c["d1"] // 2), c["d0"] * row
        moved = half * (8 + 2 * row * e)                                 # gather
        moved += half * (8 + row * e) + (c["d0"] * c["d1"] - half) * row * e + n * e   # scatter: the rows that stay, the updates, the result
        moved += 2 * e * (n // c["d3"] * (c["d3"] - c["d3"] // 2)) + 2 * e * (n // c["d1"] * (c["d1"] // 2))  # slices
        moved += 3 * 2 * n * e + 2 * (n + shared) * e + (n + shared) * e  # transposes, concat, expand
        return {"bytes": moved, "flops": 0}
    return {"bytes": sum(p[0] for p in passes), "flops": sum(p[1] for p in passes)}


def tolerance(case):
    kind = case["kind"]
    if kind == "layout":
        return "exact"
    if kind in ("decode", "prefill", "layer"):
        return {"rel": 1e-4}  # the bar the framework states for end-to-end logits
    if kind == "matmul":
        # fp32 through three TF32 products whose accumulator is truncated once per step of K; fp16: one rounding of the result
        return {"rel": 1e-5 + 4e-9 * case["k"]} if case["dtype"] == F32 else {"rel": 5e-4}
    return {"rel": 1e-5 if case.get("dtype", F32) == F32 else 1e-3}
