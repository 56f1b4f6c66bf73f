"""A few rows over Q4_K weights of up to 32768 inputs (csrc/gemm_ring.cu): staged rows where they fit shared memory, fetched ones where they
do not, at the sizes where the room beside them runs out.

Bar: the order of the fp32 sums over blocks is all that differs from a call of one row: 1e-5, as for the other kernels of the format."""
import numpy as np
import pytest

from conftest import rel_err_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [11008, 14336, 20480, 21504, 22016, 22528, 23040, 23808, 24064, 32768])
@pytest.mark.parametrize("m", [3, 8])
def test_long_rows(gpu, cols, m):
    w = gpu.Weight.synth("Q4_K", 1024, cols, seed=5, std=0.02)
    x = np.random.default_rng(cols + m).standard_normal((m, cols)).astype(np.float32)
    rel_err_ok(gpu.matmul_host(w, x), np.stack([gpu.matmul_host(w, r) for r in x]), 1e-5)
    w.free()
