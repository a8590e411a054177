"""The row walks of the bilinear backward at up-scales (bilinear_backward_walk.cu): against the oracle's scatter
kernel at the edges of their tiles. NHWC adds the scatter's products in its order: the same bits. NCHW sums rows first:
a sum of n terms of magnitude m is off by at most n * 2^-24 * m, here n <= 400 terms of weight sum 1 per axis step."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.float16, torch.bfloat16]


def _grads(shape, dtype, seed):
    g = torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)
    return g, g.float().numpy()


def _close(got, ref, dtype):
    got = got.float().cpu().numpy()
    scale = max(1.0, float(np.abs(ref).max()))
    rel = {torch.float32: 1e-5, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    np.testing.assert_allclose(got, ref, rtol=rel, atol=(2e-6 if dtype == torch.float32 else rel * 1e-2) * scale)


NCHW = [
    # N, C, Hin, Win, Hout, Wout
    (1, 1, 1, 1, 9, 7),        # one grad_input element
    (1, 3, 5, 6, 5, 7),        # one axis unchanged, scale barely below 1
    (2, 5, 7, 13, 13, 25),     # 2h - 1: odd rows, one column per thread short of two
    (3, 7, 25, 21, 50, 42),    # 2x with rows that are no multiple of 4
    (1, 2, 65, 65, 513, 513),  # eight times: lanes share a sum, bands split the rows
    (1, 1, 3, 50, 40, 1300),   # a factor of 26 at which grads of four bytes do not fit a block: the kernel without a walk
    (1, 1, 2, 9, 3, 3000),     # a factor of 333 along the row
    (40, 9, 3, 4, 5, 7),       # many planes per block, a partial last group
    (1, 1, 300, 2, 301, 3),    # long columns, narrow rows
    (1, 1, 2, 3, 2, 5000),     # a row too long for the walk: the direct kernel
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("align", [False, True])
@pytest.mark.parametrize("shape", NCHW)
def test_nchw_columns(ops, oracle, dev, dtype, align, shape):
    n, c, hi, wi, ho, wo = shape
    g, g32 = _grads((n, c, ho, wo), dtype, 7)
    ref = oracle.bilinear2d_bwd(g32, (hi, wi), align)
    _close(ops.upsample_bilinear2d_backward(g.to(dev), (ho, wo), (n, c, hi, wi), align), ref, dtype)
    # the same grads one element into a buffer: no 16-byte alignment, copies that end at both ends of the tensor
    buf = torch.empty(g.numel() + 1, dtype=dtype, device=dev)
    view = buf[1:].view(g.shape)
    view.copy_(g)
    _close(ops.upsample_bilinear2d_backward(view, (ho, wo), (n, c, hi, wi), align), ref, dtype)


NHWC = [
    (1, 8, 1, 1, 6, 5),
    (2, 16, 9, 11, 18, 22),    # 2x: four taps per column, five at the second, three at the ends
    (1, 264, 6, 5, 11, 9),     # two slices of the channels, the second one partly filled in 16-bit types
    (3, 8, 7, 40, 29, 133),    # nine taps and more per column
    (1, 48, 70, 3, 139, 7),    # bands of rows
    (70, 8, 2, 3, 4, 5),       # several images per block, a partial last group
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("align", [False, True])
@pytest.mark.parametrize("shape", NHWC)
def test_nhwc_walk_has_the_bits_of_the_scatter(ops, oracle, dev, dtype, align, shape):
    n, c, hi, wi, ho, wo = shape
    g, g32 = _grads((n, ho, wo, c), dtype, 8)
    got = ops.upsample_bilinear2d_backward(g.to(dev), (ho, wo), (n, hi, wi, c), align, "NHWC")
    ref = torch.from_numpy(oracle.bilinear2d_bwd(g32, (hi, wi), align, fmt=oracle.NHWC)).to(dtype)
    assert torch.equal(got.cpu(), ref)


@pytest.mark.parametrize("fmt", ["NCHW", "NHWC"])
@pytest.mark.parametrize("align", [False, True])
@pytest.mark.parametrize("shape", [(2, 8, 6, 9, 13, 19), (1, 8, 5, 7, 40, 55)])
def test_nonfinite_grads(ops, oracle, dev, fmt, align, shape):
    """Zero weights at clamped borders are real products: an Inf there gives NaN, as in the scatter."""
    n, c, hi, wi, ho, wo = shape
    full = (n, ho, wo, c) if fmt == "NHWC" else (n, c, ho, wo)
    g, g32 = _grads(full, torch.float32, 9)
    flat = g.view(-1)
    for k, i in enumerate([0, flat.numel() - 1, flat.numel() // 3, flat.numel() // 2 + 5]):
        flat[i] = [float("inf"), float("-inf"), float("nan")][k % 3]
    g32 = g.numpy()
    in_size = (n, hi, wi, c) if fmt == "NHWC" else (n, c, hi, wi)
    got = ops.upsample_bilinear2d_backward(g.to(dev), (ho, wo), in_size, align, fmt).cpu().numpy()
    ref = oracle.bilinear2d_bwd(g32, (hi, wi), align, fmt=getattr(oracle, fmt))
    for test in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(test(got), test(ref))


# (shape, columns per thread, planes per block): every instantiation, one block per SM, few planes for want of shared memory
REACHED = [((2, 3, 5, 40, 9, 45), 1, 5), ((3, 5, 9, 30, 20, 70), 2, 7), ((1, 1, 10, 500, 20, 1000), 2, 1),
           ((2, 1, 20, 900, 40, 1800), 4, 1), ((1, 2, 8, 225, 13, 337), 1, 1), ((1, 2, 20, 30, 37, 88), 2, 2), ((1, 2, 4, 1500, 9, 4000), 8, 1), ((1, 1, 3, 2000, 5, 4096), 8, 1),
           ((1, 2, 33, 65, 260, 520), 4, 1), ((2, 3, 16, 16, 256, 256), 4, 1)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("align", [False, True])
@pytest.mark.parametrize("shape,per_thread,planes", REACHED)
def test_nchw_columns_are_reached(ops, oracle, dev, dtype, align, shape, per_thread, planes):
    n, c, hi, wi, ho, wo = shape
    plan = ops.debug_plan("bilinear_backward_walk", 4 if dtype == torch.float32 else 2, shape, "NCHW", align)
    assert plan is not None and plan[4] == per_thread and planes <= plan[5] <= max(planes, 4)
    g, g32 = _grads((n, c, ho, wo), dtype, 10)
    got = ops.upsample_bilinear2d_backward(g.to(dev), (ho, wo), (n, c, hi, wi), align)
    _close(got, oracle.bilinear2d_bwd(g32, (hi, wi), align), dtype)


@pytest.mark.parametrize("fmt", ["NCHW", "NHWC"])
@pytest.mark.parametrize("scale,taken", [(2.2, False), (2.4, True), (2.5, True), (2.7, True), (4.0, True)])
def test_user_scales(ops, oracle, dev, fmt, scale, taken):
    """Scales that run past the input pile grads up on its last row and column: to the other kernels; smaller steps than the
    extents suggest leave the last rows and columns without grads."""
    n, c, hi, wi, ho, wo = 2, 8, 24, 20, 60, 50
    plan = ops.debug_plan("bilinear_backward_walk", 4, (n, c, hi, wi, ho, wo), fmt, False, (scale, scale))
    assert (plan is not None) == taken
    full, size = ((n, ho, wo, c), (n, hi, wi, c)) if fmt == "NHWC" else ((n, c, ho, wo), (n, c, hi, wi))
    g, g32 = _grads(full, torch.float32, 11)
    got = ops.upsample_bilinear2d_backward(g.to(dev), (ho, wo), size, False, fmt, scales=(scale, scale))
    ref = oracle.bilinear2d_bwd(g32, (hi, wi), False, (scale, scale), fmt=getattr(oracle, fmt))
    _close(got, ref, torch.float32)


@pytest.mark.parametrize("fmt,c,hi,ho", [("NHWC", 48, 5000, 12001), ("NCHW", 3, 5000, 12001), ("NHWC", 8, 5000, 9001)])
def test_tall_planes(ops, oracle, dev, fmt, c, hi, ho):
    """More than 64 bands, and the narrow image that the gather kernel serves."""
    plan = ops.debug_plan("bilinear_backward_walk", 4, (1, c, hi, 5, ho, 9), fmt)
    assert plan is None if c == 8 else -(-hi // plan[0]) > 64
    full, size = ((1, ho, 9, c), (1, hi, 5, c)) if fmt == "NHWC" else ((1, c, ho, 9), (1, c, hi, 5))
    g, g32 = _grads(full, torch.float32, 12)
    got = ops.upsample_bilinear2d_backward(g.to(dev), (ho, 9), size, False, fmt)
    _close(got, oracle.bilinear2d_bwd(g32, (hi, 5), False, fmt=getattr(oracle, fmt)), torch.float32)
