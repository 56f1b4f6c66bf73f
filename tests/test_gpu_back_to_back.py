"""Calls queued on a stream without a pause, each with data of its own, through the stream's one scratch: every launch starts while those before
it still run, and none may see what an earlier call left in the scratch. Each result equals that of the same call made alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def alone_then_queued(gpu, calls, size):
    """calls[i](out pointer) each made with the GPU idle, then all of them queued, several times over."""
    alone, outs = [], [gpu.DeviceBuffer(4 * size) for _ in calls]
    for call, out in zip(calls, outs):
        call(out.ptr)
        gpu.sync()
        alone.append(out.download(np.float32, size).copy())
    assert len({a.tobytes() for a in alone}) == len(calls)
    for _ in range(8):
        for call, out in zip(calls, outs):
            call(out.ptr)
    for out, want in zip(outs, alone):
        assert np.array_equal(out.download(np.float32, size), want)


@pytest.mark.parametrize("dim,heads,group,keys,bits", [(128, 1, 1, 300, 4), (128, 2, 4, 700, 3), (64, 1, 8, 1000, 2), (64, 2, 1, 600, 8)])
def test_attention_over_blocks(gpu, dim, heads, group, keys, bits):
    from skainet_b200.kvstore import DeviceKvCacheStore, TurboQuantConfig
    rng = np.random.default_rng(keys)
    c = TurboQuantConfig.polarOnly(bits)
    store = DeviceKvCacheStore(3, heads, dim, keys, keyConfig=c, valueConfig=c)
    rows = [[rng.standard_normal((keys, heads, dim)).astype(np.float32) for _ in range(2)] for _ in range(3)]
    for p in range(keys):
        for layer in range(3):
            store.appendToken(layer, rows[layer][0][p], rows[layer][1][p])
    qs = [gpu.DeviceBuffer.from_host(rng.standard_normal((heads * group, dim)).astype(np.float32)) for _ in range(2)]
    calls = [lambda out, layer=layer, q=q: store.decodeStep(layer, q.ptr, out, heads * group, 0, keys) for q in qs for layer in range(3)]
    alone_then_queued(gpu, calls, heads * group * dim)
    store.free()


@pytest.mark.parametrize("batch,kv_heads,group,dim,context", [(1, 1, 4, 128, 900), (2, 2, 1, 64, 600), (3, 1, 8, 64, 2000)])
def test_decode_attention(gpu, batch, kv_heads, group, dim, context):
    rng = np.random.default_rng(context)
    lens = gpu.DeviceBuffer.from_host(np.full(batch, context, np.int32))
    caches = [[gpu.DeviceBuffer.from_host(rng.standard_normal((batch, kv_heads, context, dim)).astype(np.float16)) for _ in range(2)] for _ in range(3)]
    qs = [gpu.DeviceBuffer.from_host(rng.standard_normal((batch, kv_heads * group, dim)).astype(np.float32)) for _ in range(2)]
    calls = [lambda out, k=k, v=v, q=q: gpu.attn_decode(q.ptr, k.ptr, v.ptr, out, batch, kv_heads * group, kv_heads, dim, context, lens.ptr, context, float(dim ** -0.5))
             for q in qs for k, v in caches]
    alone_then_queued(gpu, calls, batch * kv_heads * group * dim)


@pytest.mark.parametrize("enc,rows,cols,m", [("Q4_K", 600, 512, 1), ("Q4_K", 4096, 1024, 2), ("Q4_K", 2048, 512, 6), ("Q4_K", 1000, 768, 12), ("Q8_0", 700, 512, 1),
                                             ("Q8_0", 512, 512, 5), ("Q6_K", 600, 512, 3), ("Q6_K", 600, 512, 20), ("Q5_K", 600, 512, 2)])
def test_linears(gpu, enc, rows, cols, m):
    rng = np.random.default_rng(rows + m)
    bytes_per = {"Q4_K": 144, "Q8_0": 34, "Q6_K": 210, "Q5_K": 176}[enc]
    raw = rng.integers(0, 256, (rows, cols // (32 if enc == "Q8_0" else 256), bytes_per)).astype(np.uint8)
    for at in {"Q4_K": (1, 3), "Q8_0": (1,), "Q6_K": (209,), "Q5_K": (1, 3)}[enc]:
        raw[:, :, at] = 0x20                                   # binary16 factors of about 2^-7
    w = gpu.Weight.upload(raw.reshape(-1), enc, rows, cols)
    xs = [gpu.DeviceBuffer.from_host(((10.0 ** (j % 3)) * rng.standard_normal((m, cols))).astype(np.float32)) for j in range(6)]
    alone_then_queued(gpu, [lambda out, x=x: gpu.matmul(w, x.ptr, m, out) for x in xs], m * rows)
    w.free()
