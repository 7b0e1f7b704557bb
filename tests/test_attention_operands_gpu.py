"""Attention chains of a graph whose operands lie where the kernels cannot read them as they are."""
import numpy as np
import pytest

from rmlk_b200.graphspec import GraphSpec

pytestmark = pytest.mark.gpu


def i64(*v):
    return np.array(v, np.int64)


def attention_graph(KV, G, D, project=0):
    g = GraphSpec()
    H = KV * G
    g.input("q", np.float32, [0, H, 0, D])
    for name in ("new_k", "new_v", "past_k", "past_v"):
        g.input(name, np.float32, [0, KV, 0, D])
    g.input("mask", np.float32, [0, 1, 0, 0])
    g.const("scale", np.array(D ** -0.5, np.float32))
    g.const("ax2", i64(2))
    g.const("rep", i64(1, 1, G, 1, 1))
    g.const("heads", i64(0, H, -1, D))
    g.op("Concat", ["past_k", "new_k"], "present_k", axis=2)
    g.op("Concat", ["past_v", "new_v"], "present_v", axis=2)

    def heads(c):
        return g.op("Reshape", [g.op("Expand", [g.op("Unsqueeze", [c, "ax2"]), "rep"]), "heads"])

    sc = g.op("MatMul", ["q", g.op("Transpose", [heads("present_k")], perm=[0, 1, 3, 2])])
    pr = g.op("Softmax", [g.op("Add", [g.op("Mul", [sc, "scale"]), "mask"])], axis=-1)
    ctx = g.op("MatMul", [pr, heads("present_v")], "ctx")
    if project:
        g.const("w", (np.random.default_rng(2).standard_normal((H * D, project)) * 0.05).astype(np.float32))
        g.const("rows", i64(0, 0, H * D))
        g.op("MatMul", [g.op("Reshape", [g.op("Transpose", [ctx], perm=[0, 2, 1, 3]), "rows"]), "w"], "y")
        g.output("y")
    else:
        g.output("ctx")
    for o in ("present_k", "present_v"):
        g.output(o)
    return g


# one token as fp32 and as pairs of f16, several tokens
@pytest.mark.parametrize("B,S,project", [(2, 1, 0), (6, 1, 96), (2, 5, 0), (2, 5, 96)])
def test_queries_off_16_byte_boundaries(cuda, B, S, project):
    import torch
    from oracle import graph_cpu
    from rmlk_b200 import dtypes as dt
    from rmlk_b200.runtime import ModelInstance
    KV, G, D, T = 2, 4, 64, 70
    g = attention_graph(KV, G, D, project)
    inst = ModelInstance(g.to_runtime())
    inst.bind("present_k", "past_k")
    inst.bind("present_v", "past_v")
    r = np.random.default_rng(S)
    feeds = {"q": r.standard_normal((B, KV * G, S, D), dtype=np.float32), "new_k": r.standard_normal((B, KV, S, D), dtype=np.float32),
             "new_v": r.standard_normal((B, KV, S, D), dtype=np.float32), "past_k": r.standard_normal((B, KV, T, D), dtype=np.float32),
             "past_v": r.standard_normal((B, KV, T, D), dtype=np.float32), "mask": np.zeros((B, 1, S, T + S), np.float32)}
    store = torch.zeros(feeds["q"].size + 1, device=cuda)
    store[1:] = torch.from_numpy(feeds["q"]).to(cuda).flatten()
    for n, x in feeds.items():
        if n != "q":
            inst.set_input(n, x)
    inst.set_input_ptr("q", dt.F32, list(feeds["q"].shape), store.data_ptr() + 4, True)
    torch.cuda.synchronize()
    inst.launch()
    name = "y" if project else "ctx"
    got, want = inst.read(name), graph_cpu.run_graph(g, feeds)[name]
    assert np.max(np.abs(got - want)) <= 1e-4 * np.max(np.abs(want))


# requests, new tokens, keys in the cache, one launch: few rows behind a long cache are shared out over the GPU by the single operators
@pytest.mark.parametrize("B,S,T,one", [(1, 2, 600, False), (1, 16, 2000, False), (4, 4, 64, False), (1, 30, 90, True), (2, 64, 64, True), (8, 100, 30, True),
                                       (8, 33, 1100, True)])
def test_tokens_behind_a_cache(cuda, B, S, T, one):
    import os
    from rmlk_b200.runtime import ModelInstance
    KV, G, D = 8, 4, 64
    g = attention_graph(KV, G, D)
    fused = ModelInstance(g.to_runtime())
    os.environ["RMLK_B200_ATTENTION"] = "0"
    try:
        single = ModelInstance(g.to_runtime())
    finally:
        del os.environ["RMLK_B200_ATTENTION"]
    r = np.random.default_rng(S)
    feeds = {"q": r.standard_normal((B, KV * G, S, D), dtype=np.float32), "new_k": r.standard_normal((B, KV, S, D), dtype=np.float32),
             "new_v": r.standard_normal((B, KV, S, D), dtype=np.float32), "past_k": r.standard_normal((B, KV, T, D), dtype=np.float32),
             "past_v": r.standard_normal((B, KV, T, D), dtype=np.float32), "mask": np.zeros((B, 1, S, T + S), np.float32)}
    outs = []
    for inst in (fused, single):
        inst.bind("present_k", "past_k")
        inst.bind("present_v", "past_v")
        outs.append(inst.run(feeds)["ctx"])
    assert np.max(np.abs(outs[0] - outs[1])) <= 1e-5 * np.max(np.abs(outs[1]))
    assert (fused.last_launches < single.last_launches) == one
