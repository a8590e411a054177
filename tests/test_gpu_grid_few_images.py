"""2-D grid sampler backward with few images, where the staged kernels take fewer channels per block: both modes against the
CPU oracle at channel counts that leave a last group partly filled. Bars as for the other grid-sampler tests: sums in
another order, rtol 1e-5 with the absolute term scaled by the largest magnitude."""
import numpy as np
import pytest
import torch

from test_gpu_parity import gen, quant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("shape", [(1, 100, 9, 11, 13, 10), (1, 303, 6, 7, 9, 8), (2, 77, 8, 8, 16, 5), (1, 256, 5, 4, 7, 9)])
def test_few_images(ops, oracle, dev, dtype, deterministic, shape):
    n, c, h, w, ho, wo = shape
    x, x32 = quant(torch.randn((n, c, h, w), generator=gen(160)), dtype)
    grid, g32 = quant(torch.rand((n, ho, wo, 2), generator=gen(161)) * 2.2 - 1.1, dtype)
    go, go32 = quant(torch.randn((n, c, ho, wo), generator=gen(162)), dtype)
    ops.set_deterministic(deterministic)
    try:
        gi, gg = ops.grid_sampler2d_backward(go.to(dev), x.to(dev), grid.to(dev), 0, 0, False)
    finally:
        ops.set_deterministic(False)
    ri, rg = oracle.grid_sampler2d_bwd(go32, x32, g32, 0, 0, False)
    ulp = 0.0 if dtype == torch.float32 else 2.0 ** -11
    for got, ref in ((gi, ri), (gg, rg)):
        got = got.float().cpu().numpy()
        bar = (1e-5 + ulp) * np.abs(ref) + 2e-6 * max(1.0, float(np.abs(ref).max())) + (2.0 ** -25 if ulp else 0.0)
        assert (np.abs(got - ref) <= bar).all(), float((np.abs(got - ref) - bar).max())
