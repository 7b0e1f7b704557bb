"""fp32 products on pairs of f16 whose rows or columns span more than one scale holds: as accurate as where every element has its own exponent."""
import numpy as np
import pytest

from rmlk_b200.graphspec import GraphSpec

pytestmark = pytest.mark.gpu

LOWEST = float(np.finfo(np.float32).min)


def _check(a, b, got, extra=0.0):
    """float64 operands: 2^-21 for what the operands are held to, one truncated fp32 addition per 16 products; `extra`: what the rows themselves may be off by"""
    want, mag = a @ b, abs(a) @ abs(b)
    bound = mag * (2.0 ** -20 + 2.0 ** -23 * (a.shape[1] / 16 + 2) + extra) + 2.0 ** -140
    off = abs(got - want)
    assert bool((off <= bound).all()), float((off / bound).max())


# the tiles that take one scale per row and those that take several chunks, K splits, sizes that are padded
@pytest.mark.parametrize("m,n,k", [(256, 128, 64), (300, 200, 777), (256, 384, 4096), (1030, 2048, 512)])
@pytest.mark.parametrize("big", [2.0 ** 27, 2.0 ** 30, 2.0 ** 40, 2.0 ** 52, 2.0 ** 100, LOWEST])
@pytest.mark.parametrize("which", ["table", "rows", "both"])
def test_lookups(cuda, m, n, k, big, which):
    """One-hot rows read a table with one huge entry in every column; an identity reads rows with one huge value; both sparse."""
    import torch
    from rmlk_b200 import kernels as K
    gen = torch.Generator(device=cuda)
    gen.manual_seed(m + k)
    rows, cols = torch.arange(m, device=cuda), torch.arange(n, device=cuda)

    def pick(count, of):
        return torch.randint(0, of, (count,), device=cuda, generator=gen)

    if which == "table":
        a = torch.zeros(m, k, device=cuda)
        a[rows, pick(m, k)] = 1.0
        b = torch.randn(k, n, device=cuda, generator=gen)
        b[pick(n, k), cols] = big
    elif which == "rows":
        a = torch.randn(m, k, device=cuda, generator=gen)
        a[rows, pick(m, k)] = big
        b = torch.zeros(k, n, device=cuda)
        b[pick(n, k), cols] = 1.0
    else:
        a, b = torch.randn(m, k, device=cuda, generator=gen), torch.randn(k, n, device=cuda, generator=gen)
        a[:, k // 2:] *= 2.0 ** -40
        b[: k // 2] *= 0.0
        b[k // 2:] *= 2.0 ** -20
        b[pick(n, k // 2), cols] = big * 2.0 ** -40 if big > 0 else 2.0 ** 60
        a[:, : k // 2] *= (torch.rand(m, k // 2, device=cuda, generator=gen) < 2.0 / k).float()
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    _check(a.double(), b.double(), K.matmul(a, b, workspace=ws).double())


def test_every_exponent(cuda):
    import torch
    from rmlk_b200 import kernels as K
    m, n, k = 300, 260, 500
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)

    def spread(*shape):
        x = torch.randn(*shape, device=cuda, generator=gen) * torch.exp2(torch.randint(-60, 61, shape, device=cuda, generator=gen).float())
        return x * (torch.rand(*shape, device=cuda, generator=gen) < 0.1)

    a, b = spread(m, k), spread(k, n)
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    _check(a.double(), b.double(), K.matmul(a, b, workspace=ws).double())


# constant tables: a single one, blocks of a merged product, blocks of columns that are sent to the host one by one
@pytest.mark.parametrize("rows", [5, 8, 64, 300])
@pytest.mark.parametrize("big", [2.0 ** 40, LOWEST])
def test_constant_tables(cuda, rows, big):
    import torch
    from rmlk_b200.runtime import ModelInstance
    K, r = 640, np.random.default_rng(rows)
    sizes = {"a": 128, "b": 96, "c": 260, "wide": 148 * 128 * 2}
    g = GraphSpec()
    g.input("x", np.float32, [0, K])
    tables = {}
    for name, n in sizes.items():
        t = r.standard_normal((K, n), dtype=np.float32)
        t[r.integers(0, K, n), np.arange(n)] = big
        tables[name] = t
        g.const("w_" + name, t)
    for name in ("a", "b", "c"):
        g.op("Neg", [g.op("MatMul", ["x", "w_" + name])], name)
    g.op("MatMul", ["x", "w_wide"], "wide")
    for name in sizes:
        g.output(name)
    inst = ModelInstance(g.to_runtime())
    x = np.zeros((rows, K), np.float32)
    x[np.arange(rows), r.integers(0, K, rows)] = 1.0
    host = torch.empty(rows, sizes["wide"], pin_memory=True)
    for streamed in (False, True):
        if streamed:
            inst.stream_output("wide", host.data_ptr(), host.numel() * 4)
        inst.set_input("x", x)
        inst.launch()
        inst.wait_outputs()
        got = {n: inst.read(n) for n in sizes}
        if streamed:
            got["wide"] = host.numpy()
        for n in sizes:
            _check(x.astype(np.float64), tables[n].astype(np.float64), got[n] * (1.0 if n == "wide" else -1.0))


def _selection(r, k, n):
    """[k, n] with one 1 in every column"""
    w = np.zeros((k, n), np.float32)
    w[r.integers(0, k, n), np.arange(n)] = 1.0
    return w


# rows that RMSNorm and SwiGLU hand over as pairs: a few wide CTAs, many rows; products that leave the range of fp32 on the way
@pytest.mark.parametrize("rows,cols", [(5, 64), (64, 2048), (600, 2048), (7, 4096), (600, 4096)])
@pytest.mark.parametrize("case", ["weights", "values", "tiny", "overflow"])
def test_rmsnorm_rows(cuda, rows, cols, case):
    from rmlk_b200.runtime import ModelInstance
    r = np.random.default_rng(cols)
    x, w = r.standard_normal((rows, cols), dtype=np.float32), r.standard_normal(cols, dtype=np.float32)
    if case == "weights":
        w[r.integers(0, cols, 3)] = 2.0 ** 60
    elif case == "values":
        x[:, ::3] *= 2.0 ** -50
    elif case == "tiny":
        x *= 2.0 ** -70
        w *= 2.0 ** -70
        x[:, 1] *= 2.0 ** 40
    else:
        x *= 2.0 ** 50
        w *= 2.0 ** 77
        w[::5] = 1.0
    sel = _selection(r, cols, 192)
    g = GraphSpec()
    g.input("x", np.float32, [0, cols])
    g.const("two", np.array(2.0, np.float32))
    g.const("eps", np.array(1e-5, np.float32))
    g.const("w", w)
    g.const("sel", sel)
    mean = g.op("ReduceMean", [g.op("Pow", ["x", "two"])], axes=[-1], keepdims=1)
    y = g.op("Mul", [g.op("Div", ["x", g.op("Sqrt", [g.op("Add", [mean, "eps"])])]), "w"])
    g.op("MatMul", [y, "sel"], "out")
    g.output("out")
    got = ModelInstance(g.to_runtime()).run({"x": x})["out"]
    x64 = x.astype(np.float64)
    y64 = x64 / np.sqrt((x64 ** 2).mean(-1, keepdims=True) + np.float64(np.float32(1e-5))) * w
    _check(y64, sel.astype(np.float64), got, extra=1e-6)


@pytest.mark.parametrize("rows,cols", [(5, 128), (64, 8192), (600, 2048), (9, 16384)])
def test_swiglu_rows(cuda, rows, cols):
    """Gates far below zero: values from 1 down to 1e-40 in a row."""
    from rmlk_b200.runtime import ModelInstance
    r = np.random.default_rng(cols)
    gate = (r.standard_normal((rows, cols)) * 30).astype(np.float32)
    up = r.standard_normal((rows, cols), dtype=np.float32)
    sel = _selection(r, cols, 192)
    g = GraphSpec()
    g.input("gate", np.float32, [0, cols])
    g.input("up", np.float32, [0, cols])
    g.const("sel", sel)
    g.op("MatMul", [g.op("Mul", [g.op("Mul", ["gate", g.op("Sigmoid", ["gate"])]), "up"]), "sel"], "out")
    g.output("out")
    got = ModelInstance(g.to_runtime()).run({"gate": gate, "up": up})["out"]
    g64 = gate.astype(np.float64)
    act = g64 / (1 + np.exp(-g64)) * up
    # (1 / (1 + exp(-g)) underflows in fp32 from g = -88 on)
    off, bound = np.abs(got - act @ sel), (np.abs(act) @ sel) * (2.0 ** -20 + 2.0 ** -23 * (cols / 16 + 2) + 2e-6) + 2.0 ** -118
    assert (off <= bound).all(), float((off / bound).max())


@pytest.mark.parametrize("B,T", [(5, 40), (64, 300)])
def test_attention_rows(cuda, B, T):
    """The result of one-token attention as pairs: value dims of very different size, some KV heads only."""
    from rmlk_b200.runtime import ModelInstance
    from test_attention_operands_gpu import attention_graph
    KV, G, D = 4, 4, 64
    H = KV * G
    r = np.random.default_rng(B)
    sel = _selection(r, H * D, 96)
    g = attention_graph(KV, G, D, project=96)
    g.constants["w"] = sel
    inst = ModelInstance(g.to_runtime())
    inst.bind("present_k", "past_k")
    inst.bind("present_v", "past_v")
    feeds = {"q": r.standard_normal((B, H, 1, D), dtype=np.float32), "new_k": r.standard_normal((B, KV, 1, D), dtype=np.float32),
             "new_v": r.standard_normal((B, KV, 1, D), dtype=np.float32), "past_k": r.standard_normal((B, KV, T, D), dtype=np.float32),
             "past_v": r.standard_normal((B, KV, T, D), dtype=np.float32), "mask": np.zeros((B, 1, 1, T + 1), np.float32)}
    for n in ("new_v", "past_v"):
        feeds[n][:, 1, :, 5] *= np.float32(2.0 ** 60)
        feeds[n][:, 2, :, ::2] *= np.float32(2.0 ** -45)
    got = inst.run(feeds)["y"]
    k = np.concatenate([feeds["past_k"], feeds["new_k"]], 2).astype(np.float64).repeat(G, 1)
    v = np.concatenate([feeds["past_v"], feeds["new_v"]], 2).astype(np.float64).repeat(G, 1)
    s = feeds["q"].astype(np.float64) @ k.transpose(0, 1, 3, 2) * np.float64(np.float32(D ** -0.5))
    e = np.exp(s - s.max(-1, keepdims=True))
    p = e / e.sum(-1, keepdims=True)
    want, mag = (p @ v).reshape(B, H * D) @ sel, (p @ np.abs(v)).reshape(B, H * D) @ sel
    assert (np.abs(got[:, 0] - want) <= 2e-5 * mag).all()


def _attention_cases():
    def value_behind(q, k, v):  # a finite, very large value at a key that the later rows see and the earlier ones do not
        v[0, 0, 100] = 1e30
        v[0, 1, 101, 7] = LOWEST

    def values_apart(q, k, v):  # blocks of values 2^60 apart, dims 2^45 apart
        v[:, 0, 64:128] *= 2.0 ** 60
        v[:, 1, :, ::3] *= 2.0 ** -45

    def faint_giant(q, k, v):  # a huge value under a weight of 2^-50 beside ordinary ones under weights of 1
        k[:, :, 5] = 0
        q[:, :, :, :, 0] = 8.0
        k[:, :, :, 0] = 0
        k[:, :, 5, 0] = -35.0
        v[:, :, 5] *= 2.0 ** 45

    def keys_apart(q, k, v):  # scores far beyond what one scale for queries and keys holds
        k[0, 0, 30] *= 1e20
        q[0, 1, 0, 9] *= 1e12

    def query_apart(q, k, v):  # one row of the tile 2^60 above the others, with scores of ordinary size
        q[:, :, :, 3] *= 2.0 ** 60
        q[:, :, :, 3, 1:] = 0
        k[:, :, :, 0] *= 2.0 ** -60
        q[:, :, :, 4:, 1:] *= 4.0

    return {f.__name__: f for f in (value_behind, values_apart, faint_giant, keys_apart, query_apart)}


@pytest.mark.parametrize("case", sorted(_attention_cases()))
@pytest.mark.parametrize("B,KV,G,S", [(1, 2, 1, 130), (1, 2, 4, 150)])
def test_prompt_attention(cuda, case, B, KV, G, S):
    import torch
    from rmlk_b200 import kernels as K
    gen = torch.Generator(device=cuda)
    gen.manual_seed(S)
    q, k, v = (torch.randn(B, KV, *x, 64, device=cuda, generator=gen) for x in ((G, S), (S,), (S,)))
    _attention_cases()[case](q, k, v)
    mask = torch.zeros(B, 1, S, S, device=cuda).masked_fill(torch.arange(S, device=cuda)[None] > torch.arange(S, device=cuda)[:, None], LOWEST)
    got = K.gqa_prefill_attention(q, k, v, 0.125, mask).double()
    s = torch.einsum("bkgsd,bktd->bkgst", q.double(), k.double()) * 0.125
    # (what fp32 products of this size round to: a score is off by 2^-22 of its terms, a weight by that much of itself)
    slack = (torch.einsum("bkgsd,bktd->bkgst", q.double().abs(), k.double().abs()) * 0.125 * 2.0 ** -22).amax(-1, keepdim=True)
    p = torch.softmax(s + mask.double()[:, :, None], -1)
    want = torch.einsum("bkgst,bktd->bkgsd", p, v.double())
    mag = torch.einsum("bkgst,bktd->bkgsd", p, v.double().abs()) * (2e-6 + 2 * slack.clamp(max=1.0))
    lay = lambda x: x.permute(0, 3, 1, 2, 4).reshape(B, S, KV * G, 64)  # noqa: E731
    off, bound = (got - lay(want)).abs(), lay(mag)
    settled = (lay(slack.expand_as(want)) < 0.1)  # (rows of scores beyond 2^20 are one-hot up to rounding: only that they are numbers)
    assert bool((off <= bound)[settled].all()), float((off / bound)[settled].max())
    assert bool(torch.isfinite(got).all())
