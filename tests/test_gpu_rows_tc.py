"""The integer tcgen05 tiles of Q4_K and Q6_K rows (csrc/gemm_tc.cu) where they can go wrong: tiles of 16 rows with their clusters, calls of more tiles
than the GPU has SMs (whole rounds, then the rest in clusters), and the largest sums that Q6_K blocks can hold.

Bars: Q4_K sums are exact per super-block and differ in the order of the fp32 sums (1e-5, as for the other tiles); a Q6_K row has the bits of the
row kernel."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 2, 7])
@pytest.mark.parametrize("n,k", [(1, 256), (129, 1280), (300, 4352)])
def test_tiles_of_16_rows(gpu, oracle, n, k, parts):
    parts = min(parts, k // 256)
    rng = np.random.default_rng(n + k + parts)
    w_bytes = oracle.quantize_q4k((0.02 * rng.standard_normal((n, k))).astype(np.float32))
    w = gpu.Weight.upload(w_bytes, "Q4_K", n, k)
    for m in (1, 8, 9, 16, 17):
        x = rng.standard_normal((m, k)).astype(np.float32)
        dx, dy = gpu.DeviceBuffer.from_host(x), gpu.DeviceBuffer(4 * m * n)
        gpu.q4k_rows(w, dx.ptr, m, dy.ptr, 16, parts)
        got = dy.download(np.float32, m * n).reshape(m, n)
        rel_err_ok(got, oracle.matmul("Q4_K", x, w_bytes, k, n, "rm", use_ref=oracle.ref() is not None), 1e-5)
    w.free()


@pytest.mark.parametrize("n,k,m", [(128 * 160, 1024, 40), (128 * 149 + 3, 2048, 64), (9000, 1280, 300)])
def test_more_tiles_than_sms(gpu, n, k, m):
    """Whole rounds and the clusters of the rest: every row of the batch is that of a call of eight rows."""
    rng = np.random.default_rng(n)
    w = gpu.Weight.synth("Q4_K", n, k, seed=7, std=0.02)
    x = rng.standard_normal((m, k)).astype(np.float32)
    assert gpu.q4k_rows_plan(w, m)[0] >= 64
    want = np.concatenate([gpu.matmul_host(w, x[i:i + 8]) for i in range(0, m, 8)])
    rel_err_ok(gpu.matmul_host(w, x), want, 1e-5)
    w.free()


@pytest.mark.parametrize("m", [9, 20, 64, 130])
@pytest.mark.parametrize("codes,scales", [((0, 2), (127, 128)), ((0, 2), (-128, -127)), ((62, 64), (-128, -127)), ((0, 64), (-128, 128))])
def test_q6k_extreme_blocks(gpu, m, codes, scales):
    """Codes, scales and activations at their ends, of one sign and mixed: planes and their offsets hold them, and the sums are exact."""
    n, nb, rng = 140, 3, np.random.default_rng(m)
    q = rng.integers(*codes, (n, nb, 2, 4, 32)).astype(np.uint8)
    raw = np.zeros((n, nb, 210), np.uint8)
    raw[..., :128] = np.stack([(q[..., 0, :] & 15) | ((q[..., 2, :] & 15) << 4), (q[..., 1, :] & 15) | ((q[..., 3, :] & 15) << 4)], -2).reshape(n, nb, 128)
    raw[..., 128:192] = ((q[..., 0, :] >> 4) | ((q[..., 1, :] >> 4) << 2) | ((q[..., 2, :] >> 4) << 4) | ((q[..., 3, :] >> 4) << 6)).reshape(n, nb, 64)
    raw[..., 192:208] = rng.integers(*scales, (n, nb, 16)).astype(np.int8).view(np.uint8)
    raw[..., 208:] = np.full((n, nb, 1), 2.0 ** -12, np.float16).view(np.uint8)
    x = rng.integers(126, 128, (m, nb * 256)).astype(np.float32)
    x[1::2] *= rng.choice([-1.0, 1.0], (x[1::2].shape))
    x[2::4] *= -1.0
    w = gpu.Weight.upload(raw.reshape(-1), "Q6_K", n, 256 * nb)
    got = gpu.matmul_host(w, x)
    for i in (0, 1, 2, m // 2, m - 1):
        assert np.array_equal(got[i], gpu.matmul_host(w, x[i:i + 1])[0])
    w.free()
