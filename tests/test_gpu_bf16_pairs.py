"""BF16 linears of many rows on pairs of SMs (csrc/gemm_bf16_tc.cu) at the edges of their tiles (256 weight rows, 256 activation rows), with one step of
the contraction and with more tiles than there are pairs, beside shapes that stay with single CTAs.

Bar: products of bf16 numbers are exact in fp32, the sums run over up to 4096 of them: 1e-5 of the largest result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,m", [(256, 64, 129), (255, 64, 256), (257, 128, 257), (1, 192, 300), (2048, 1024, 2048), (3072, 1000, 513), (576, 2048, 700), (5000, 320, 1025), (4100, 4096, 255)])
def test_tile_edges(gpu, n, k, m):
    import torch
    g = torch.Generator().manual_seed(n + k + m)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).bfloat16()
    x = torch.randn(m, k, generator=g).bfloat16()
    dw = w.cuda()
    torch.cuda.synchronize()
    weight = gpu.Weight.from_device(dw.data_ptr(), 2 * n * k, "BF16", n, k)
    xs, ys = x.float().cuda(), [torch.full((m, n), float("nan"), device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    for y in ys:
        gpu.matmul(weight, xs.data_ptr(), m, y.data_ptr())
    gpu.sync()
    want = x.double().cuda() @ w.double().cuda().T
    for y in ys:
        assert (y.double() - want).abs().max() <= 1e-5 * want.abs().max()
        assert torch.equal(y, ys[0])
    weight.free()
