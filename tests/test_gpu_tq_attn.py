"""Decode attention straight from TurboQuant blocks (csrc/tq_attn.cu) against attention in 64 bits over the rows that a read of the
store returns, rounded to binary16: every code width, both head sizes, groups, windows that start and end inside a 16-key tile,
fewer keys than one tile, and more than one key split.

Bar: the kernel's rows equal the rounded read bit for bit, q and the probabilities are carried to 2^-21, exp2 and the sums are fp32:
1e-5 of the result's largest value covers a few hundred such roundings; a wrong row or sign is worth 1e-2 and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,kbits,vbits,heads,group,window", [
    (128, 4, 4, 8, 1, (0, 300)), (128, 2, 3, 2, 4, (5, 257)), (128, 3, 8, 3, 8, (0, 17)), (128, 8, 2, 1, 2, (1, 2)),
    (64, 4, 4, 4, 1, (0, 300)), (64, 3, 2, 2, 8, (7, 200)), (64, 2, 8, 1, 4, (0, 15)), (64, 8, 3, 5, 2, (130, 300))])
def test_attention_from_blocks(gpu, dim, kbits, vbits, heads, group, window):
    from skainet_b200.kvstore import DeviceKvCacheStore, TurboQuantConfig
    a, b = window
    rng = np.random.default_rng(dim + 10 * kbits + vbits)
    store = DeviceKvCacheStore(2, heads, dim, 300, keyConfig=TurboQuantConfig.polarOnly(kbits), valueConfig=TurboQuantConfig.polarOnly(vbits))
    for p in range(b):
        for layer in range(2):
            k = rng.standard_normal((heads, dim)).astype(np.float32)
            if p % 50 == 3:
                k[:, :32] = 0.0                        # a group whose scale is 0
            store.appendToken(layer, k, rng.standard_normal((heads, dim)).astype(np.float32))
    q = (3.0 * rng.standard_normal((heads * group, dim))).astype(np.float32)
    dq, dout = gpu.DeviceBuffer.from_host(q), gpu.DeviceBuffer(q.nbytes)
    store.decodeStep(1, dq.ptr, dout.ptr, heads * group, a, b)
    got = dout.download(np.float32, q.size).reshape(heads * group, dim).astype(np.float64)
    half = lambda r: np.repeat(np.asarray(r).reshape(heads, b - a, dim).astype(np.float16).astype(np.float64), group, 0)  # noqa: E731
    keys, values = half(store.readKeys(1, a, b)), half(store.readValues(1, a, b))
    score = np.einsum("hd,hnd->hn", q.astype(np.float64), keys) / np.sqrt(np.float32(dim))
    p = np.exp(score - score.max(-1, keepdims=True))
    want = np.einsum("hn,hnd->hd", p / p.sum(-1, keepdims=True), values)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    store.free()
