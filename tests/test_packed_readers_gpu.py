"""Values that a producer writes for the MatMuls behind it (pairs of f16, K slabs left unsummed): who else reads them, and in which order."""
import numpy as np
import pytest

from oracle import graph_cpu
from rmlk_b200.graphspec import GraphSpec

pytestmark = pytest.mark.gpu


def i64(*v):
    return np.array(v, np.int64)


# the one-token result of attention, [B, H, 1, D], on its way to a product: every order of B, H and D; B == H where B moves
@pytest.mark.parametrize("B,perm", [(6, (0, 2, 1, 3)), (6, (2, 0, 1, 3)), (6, (0, 1, 3, 2)), (6, (0, 3, 2, 1)), (6, (0, 3, 1, 2)), (8, (1, 0, 2, 3)), (8, (1, 2, 0, 3)),
                                    (8, (3, 2, 1, 0))])
def test_transposed_attention_result(cuda, B, perm):
    from rmlk_b200.runtime import ModelInstance
    KV, G, D, N, T = 2, 4, 64, 96, 37
    H = KV * G
    g = GraphSpec()
    g.input("q", np.float32, [0, H, 0, D])
    for name in ("new_k", "new_v", "past_k", "past_v"):
        g.input(name, np.float32, [0, KV, 0, D])
    g.input("mask", np.float32, [0, 1, 0, 0])
    r = np.random.default_rng(5)
    g.const("scale", np.array(D ** -0.5, np.float32))
    g.const("ax2", i64(2))
    g.const("rep", i64(1, 1, G, 1, 1))
    g.const("heads", i64(0, H, -1, D))
    g.const("rows", i64(B, H * D))
    g.const("w", (r.standard_normal((H * D, N)) * 0.05).astype(np.float32))
    g.op("Concat", ["past_k", "new_k"], "present_k", axis=2)
    g.op("Concat", ["past_v", "new_v"], "present_v", axis=2)

    def heads(c):
        return g.op("Reshape", [g.op("Expand", [g.op("Unsqueeze", [c, "ax2"]), "rep"]), "heads"])

    sc = g.op("MatMul", ["q", g.op("Transpose", [heads("present_k")], perm=[0, 1, 3, 2])])
    pr = g.op("Softmax", [g.op("Add", [g.op("Mul", [sc, "scale"]), "mask"])], axis=-1)
    ctx = g.op("MatMul", [pr, heads("present_v")])
    g.op("MatMul", [g.op("Reshape", [g.op("Transpose", [ctx], perm=list(perm)), "rows"]), "w"], "y")
    for o in ("y", "present_k", "present_v"):
        g.output(o)
    inst = ModelInstance(g.to_runtime())
    inst.bind("present_k", "past_k")
    inst.bind("present_v", "past_v")
    feeds = {"q": r.standard_normal((B, H, 1, D), dtype=np.float32), "new_k": r.standard_normal((B, KV, 1, D), dtype=np.float32),
             "new_v": r.standard_normal((B, KV, 1, D), dtype=np.float32), "past_k": r.standard_normal((B, KV, T, D), dtype=np.float32),
             "past_v": r.standard_normal((B, KV, T, D), dtype=np.float32), "mask": np.zeros((B, 1, 1, T + 1), np.float32)}
    got = inst.run(feeds)["y"]
    want = graph_cpu.run_graph(g, feeds)["y"]
    assert np.max(np.abs(got - want)) <= 1e-4 * np.max(np.abs(want))


# one merged product of which SwiGLU reads two blocks, and another op a third one behind it; fp32 slabs (1, 4 rows) and pairs (8, 64)
@pytest.mark.parametrize("rows", [1, 4, 8, 64])
@pytest.mark.parametrize("third_first", [False, True])
def test_third_reader_of_a_product_behind_swiglu(cuda, rows, third_first):
    from rmlk_b200.runtime import ModelInstance
    K, N = 2048, 512
    g = GraphSpec()
    g.input("x", np.float32, [0, K])
    r = np.random.default_rng(rows)
    names = ["third", "gate", "up"] if third_first else ["gate", "up", "third"]
    for n in names:
        g.const("w_" + n, (r.standard_normal((K, N)) * 0.03).astype(np.float32))
    for n in names:
        g.op("MatMul", ["x", "w_" + n], n)
    g.op("Mul", [g.op("Mul", ["gate", g.op("Sigmoid", ["gate"])]), "up"], "act")
    g.op("Neg", ["third"], "late")
    g.output("act")
    g.output("late")
    inst = ModelInstance(g.to_runtime())
    for _ in range(2):
        x = r.standard_normal((rows, K), dtype=np.float32)
        got, want = inst.run({"x": x}), graph_cpu.run_graph(g, {"x": x})
        for n in ("act", "late"):
            assert np.max(np.abs(got[n] - want[n])) <= 1e-4 * np.max(np.abs(want[n])), n
