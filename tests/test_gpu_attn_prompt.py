"""Attention of prompt rows (csrc/attention.cu: attn_prompt_kernel from 40 rows, attn_prefill_mma_kernel below) on the runtime's own
projections, against attention in 64 bits: around the 64-query and 64-key tiles, both head sizes, grouped heads,
passes that follow others (few queries over many keys, which a cluster shares, among them).

Bar: the cache rows are binary16 of the rotated keys and of the values on both sides, q and the probabilities carry 2^-21, rotation,
exp2 and sums are fp32; a rotated key whose fp32 value differs in the last place may round to another binary16 (2^-11 of it), so
2e-3 of the largest result; a wrong or missing key is worth 1e-2 and more."""
import numpy as np
import pytest

from test_gpu_llama import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,before,n", [
    (4, 4, 128, 0, 40), (8, 2, 64, 0, 39), (4, 1, 128, 0, 63), (4, 2, 128, 0, 64), (8, 8, 64, 0, 65), (2, 1, 128, 0, 129), (4, 4, 64, 0, 200), (2, 2, 128, 0, 512),
    (2, 1, 128, 500, 41), (4, 4, 64, 511, 40), (80, 10, 64, 190, 70), (2, 2, 128, 129, 64)])
def test_prompt_attention(gpu, oracle, heads, kv_heads, dim, before, n):
    from skainet_b200.llama import LlamaConfig
    cfg = LlamaConfig(1, 256, heads, kv_heads, dim, 256, 300, max_seq=600)
    m, _, _ = build(gpu, cfg, seed=n)
    tokens = np.random.default_rng(n).integers(0, cfg.vocab, size=before + n).astype(np.int32)
    width, parts = (heads + 2 * kv_heads) * dim, []
    for at, end in ((0, before), (before, before + n)):
        if end > at:
            m.forward(tokens[at:end], [end - at - 1], 0)
            parts.append(m.peek(1, (end - at) * width).reshape(end - at, -1, dim))
    qkv, got = np.concatenate(parts), m.peek(2, n * heads * dim).reshape(n, heads, dim).astype(np.float64)
    turned = np.stack([oracle.rope(qkv[p, :heads + kv_heads].copy(), heads + kv_heads, dim, p).reshape(-1, dim) for p in range(before + n)])
    q, half = turned[before:, :heads].astype(np.float64), lambda a: np.repeat(a.astype(np.float16).astype(np.float64), heads // kv_heads, 1)
    k, v = half(turned[:, heads:]), half(qkv[:, heads + kv_heads:])
    score = np.einsum("ihd,jhd->hij", q, k) / np.sqrt(dim)
    score[:, np.triu(np.ones((n, before + n), bool), before + 1)] = -np.inf
    p = np.exp(score - score.max(-1, keepdims=True))
    want = np.einsum("hij,jhd->ihd", p / p.sum(-1, keepdims=True), v)
    assert np.abs(got - want).max() <= 2e-3 * np.abs(want).max()
    m.free()
