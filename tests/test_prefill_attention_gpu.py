"""Attention of many query tokens (attention_prefill.cu) against float64."""
import pytest

pytestmark = pytest.mark.gpu


def _want(q, k, v, scale, mask):
    import torch
    B, KV, G, S, D = q.shape
    s = torch.einsum("bkgsd,bktd->bkgst", q.double(), k.double()) * scale
    if mask is not None:
        m = mask.double()
        s = s + (m.view(B, KV, G, S, -1) if m.shape[1] > 1 else m[:, :, None])
    return torch.einsum("bkgst,bktd->bkgsd", torch.softmax(s, -1), v.double()).permute(0, 3, 1, 2, 4).reshape(B, S, KV * G, D)


def _close(got, want, v):
    # scores of this size are off by 2^-21 of |q| |k| (pairs, truncated sums): weights by some 2^-18, the result by that share of the largest value
    err = (got.double() - want).abs().max()
    assert float(err) <= 1e-5 * float(v[v.isfinite()].abs().max()), float(err)


# rows of a tile (128) filled by one head, by several, and not at all; blocks of 64 keys with remainders; rows of the mask on and off 16 bytes
@pytest.mark.parametrize("B,KV,G,S,T", [(1, 1, 1, 2, 2), (2, 2, 4, 17, 17), (1, 2, 4, 32, 64), (1, 1, 4, 33, 65), (2, 1, 3, 128, 128), (1, 2, 1, 129, 200), (1, 2, 4, 187, 187),
                                       (2, 2, 4, 5, 301), (1, 1, 2, 300, 1027)])
@pytest.mark.parametrize("masked", ["none", "causal", "padded", "random"])
def test_shapes(cuda, B, KV, G, S, T, masked):
    import torch
    from rmlk_b200 import kernels as K
    gen = torch.Generator(device=cuda)
    gen.manual_seed(B + 3 * S + 7 * T)
    q = torch.randn(B, KV, G, S, 64, device=cuda, generator=gen)
    store = torch.randn(2, B, KV, T + 9, 64, device=cuda, generator=gen)  # a cache with spare room
    k, v = store[0, :, :, :T], store[1, :, :, :T]
    low = torch.finfo(torch.float32).min
    mask = None
    if masked == "random":
        mask = torch.randn(B, KV * G, S, T, device=cuda, generator=gen)
    elif masked != "none":
        hidden = torch.arange(T, device=cuda)[None] > torch.arange(T - S, T, device=cuda)[:, None]
        mask = torch.zeros(B, 1, S, T, device=cuda).masked_fill(hidden, low)
        if masked == "padded":  # left padding: whole rows of the lowest value, whose weights are all the same
            mask[0, :, :, : T // 3] = low
            if B > 1:
                mask[1, :, :, : T - 1] = low
    got = K.gqa_prefill_attention(q, k, v, 0.125, mask)
    _close(got, _want(q, k, v, 0.125, mask), v)


def test_infinite_masks_and_values(cuda):
    """-inf in the mask, NaN and infinities in keys and values that the mask hides, extreme scales: what the single operators give."""
    import torch
    from rmlk_b200 import kernels as K
    B, KV, G, S, T = 1, 2, 2, 150, 150
    q, k, v = (torch.randn(B, KV, *x, 64, device=cuda) for x in ((G, S), (T,), (T,)))
    hidden = torch.arange(T, device=cuda)[None] > torch.arange(S, device=cuda)[:, None]
    mask = torch.zeros(B, 1, S, T, device=cuda).masked_fill(hidden, float("-inf"))
    mask[:, :, 70:, :66] = float("-inf")  # first block and more of these rows
    mask[:, :, 3] = float("-inf")         # 0 / 0
    got, want = K.gqa_prefill_attention(q, k, v, 0.125, mask), _want(q, k, v, 0.125, mask)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    ok = ~torch.isnan(want)
    _close(got[ok], want[ok], v)
    mask = torch.zeros(B, 1, S, T, device=cuda).masked_fill(hidden, torch.finfo(torch.float32).min)
    v[0, 0, 140, 5] = float("nan")
    v[0, 1, 141, 6] = float("inf")
    got, want = K.gqa_prefill_attention(q, k, v, 0.125, mask), _want(q, k, v, 0.125, mask)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    big, small = q * 2.0 ** 115, k * 2.0 ** -115
    w = torch.randn_like(v)
    _close(K.gqa_prefill_attention(big, small, w, 0.125, mask), _want(q, k, w, 0.125, mask), w)


@pytest.mark.parametrize("S", [2, 33, 130])
def test_decoder_prompt(cuda, S):
    """Through the runtime: a prompt, then new tokens behind its cache, against the CPU interpreter of the graph."""
    import numpy as np
    from oracle import graph_cpu
    from rmlk_b200 import llama
    cfg = llama.LlamaConfig(hidden=256, n_heads=4, n_kv_heads=2, head_dim=64, ffn=256, vocab=131, n_layers=2)
    spec = llama.build_graph(cfg, llama.make_weights_host(cfg, seed=S))
    ids = np.random.default_rng(S).integers(0, cfg.vocab, size=(2, S + 3))
    dec = llama.Decoder(cfg, spec)
    dec.reset(2)
    past = [(np.zeros((2, cfg.n_kv_heads, 0, cfg.head_dim), np.float32),) * 2 for _ in range(cfg.n_layers)]
    for s0, s1 in [(0, S), (S, S + 2), (S + 2, S + 3)]:
        got = dec.step(ids[:, s0:s1])
        feeds = {"input_ids": ids[:, s0:s1], "attention_mask": np.ones((2, s1), np.int64),
                 "position_ids": np.broadcast_to(np.arange(s0, s1, dtype=np.int64), (2, s1 - s0)).copy()}
        for l in range(cfg.n_layers):
            feeds[f"past_key_values.{l}.key"], feeds[f"past_key_values.{l}.value"] = past[l]
        want = graph_cpu.run_graph(spec, feeds)
        past = [(want[f"present.{l}.key"], want[f"present.{l}.value"]) for l in range(cfg.n_layers)]
        assert float(np.max(np.abs(got - want["logits"])) / np.max(np.abs(want["logits"]))) <= 1e-4
