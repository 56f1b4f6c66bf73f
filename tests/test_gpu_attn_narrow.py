"""Decode attention with more (sequence, cache head) pairs than SMs (four warps a CTA, csrc/attention.cu): against attention in 64 bits over
contexts of one key, of less than one 16-key tile, of several rounds of the CTA's tiles, both head sizes, grouped heads.

Bar: q and the probabilities carry 2^-21, exp2 and sums are fp32: 1e-5 of the largest result; a lost key is worth 1e-2 and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,kv_heads,group,dim,context", [(20, 8, 4, 128, 200), (150, 1, 8, 64, 130), (40, 4, 1, 128, 17), (19, 8, 2, 64, 700)])
def test_many_pairs(gpu, batch, kv_heads, group, dim, context):
    rng = np.random.default_rng(batch)
    q = rng.standard_normal((batch, kv_heads * group, dim)).astype(np.float32)
    k, v = (rng.standard_normal((batch, kv_heads, context, dim)).astype(np.float16) for _ in range(2))
    n = rng.integers(1, context + 1, batch).astype(np.int32)
    n[0], n[1] = context, 1
    dq, dk, dv, dn = (gpu.DeviceBuffer.from_host(a) for a in (q, k, v, n))
    out = gpu.DeviceBuffer(q.nbytes)
    gpu.attn_decode(dq.ptr, dk.ptr, dv.ptr, out.ptr, batch, kv_heads * group, kv_heads, dim, context, dn.ptr, context, float(dim ** -0.5))
    got = out.download(np.float32, q.size).reshape(q.shape).astype(np.float64)
    for b in range(batch):
        kb, vb = (np.repeat(a[b, :, :n[b]].astype(np.float64), group, 0) for a in (k, v))
        s = np.einsum("hd,hnd->hn", q[b].astype(np.float64), kb) * dim ** -0.5
        p = np.exp(s - s.max(-1, keepdims=True))
        want = np.einsum("hn,hnd->hd", p / p.sum(-1, keepdims=True), vb)
        assert np.abs(got[b] - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
