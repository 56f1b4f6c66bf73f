"""Prompts through rope_prompt_kernel (csrc/llama.cu) against the CPU composer: both rotation layouts, both head sizes, grouped and
ungrouped heads, one to several CTAs a row, a pass that does not start at position 0.

Bar: that of the decoder tests (0.15 of the logits' root mean square: an int8 activation code that falls the other way travels
through the layers); a head, pair or position that is wrong is worth 1 and more."""
import numpy as np
import pytest

from test_gpu_llama import build, step_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,mode,lengths", [(4, 4, 128, 0, (9,)), (8, 2, 64, 1, (3, 14)), (16, 2, 128, 1, (1, 16)), (32, 16, 64, 0, (17,))])
def test_prompt_logits(gpu, oracle, heads, kv_heads, dim, mode, lengths):
    from skainet_b200.llama import LlamaConfig
    from oracle.llama_cpu import CpuLlama
    cfg = LlamaConfig(1, 512, heads, kv_heads, dim, 512, 300, max_seq=64, rope_mode=mode, max_batch=2)
    m, weights, gam = build(gpu, cfg, norms=True)
    tokens = np.random.default_rng(heads + dim).integers(0, cfg.vocab, size=sum(lengths)).astype(np.int32)
    cpu = CpuLlama(cfg, weights, gam)
    want = [cpu.step(int(t)) for t in tokens]
    at = 0
    for n in lengths:                                  # the second sequence: its caches and position are not the first's
        got = np.asarray(m.forward(tokens[at:at + n], list(range(n)), 1))
        for i in range(n):
            assert step_err(got[i], want[at + i]) < 0.15
        at += n
    m.free()
