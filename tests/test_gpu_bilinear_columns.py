"""The bilinear forward at widths that allow no store wider than two elements, against the CPU oracle: column groups at a
block's width and past it, a block's last column, several planes per block, and (the large plane counts) several groups per
thread. The expression tree is the oracle's, so fp32 is compared bit for bit and 16-bit results after one rounding."""
import pytest
import torch

from test_gpu_parity import DTYPES, check, gen, quant

pytestmark = pytest.mark.gpu

# (n, c, h, w, oh, ow)
SHAPES = [(1, 2, 5, 7, 13, 17), (3, 5, 9, 10, 22, 33), (1, 1, 65, 65, 200, 513), (2, 3, 4, 3, 9, 1), (1, 3, 12, 20, 31, 46),
          (1, 1, 40, 31, 17, 11), (1, 40, 60, 63, 480, 513), (2, 60, 9, 300, 80, 1025), (8, 300, 5, 9, 40, 67),
          (1, 90, 40, 31, 200, 386)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("align", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_bilinear_forward_columns(ops, oracle, dev, dtype, align, shape):
    n, c, h, w, oh, ow = shape
    x, x32 = quant(torch.randn((n, c, h, w), generator=gen(150)), dtype)
    y = ops.upsample_bilinear2d(x.to(dev), (oh, ow), align)
    check(y, oracle.bilinear2d_fwd(x32, (oh, ow), align), dtype, exact=True)
