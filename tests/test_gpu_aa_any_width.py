"""Anti-aliased down-scaling at any width and alignment: the streaming forward at every load width, the band backward with
and without parked rows, bands that hold one output row, and windows of a user scale that lie past the input.

Bars: fp32 against the oracle rtol 1e-5 / atol 1e-6 (same terms, sums split by axis: at most 25 x 25 products of weights
that sum to one, each rounding 6e-8). fp16 / bf16: half an ulp of the storage type around the oracle's fp32 value, plus the
fp32 bar."""
import numpy as np
import pytest
import torch

from test_gpu_parity import DTYPES, _poison, _same_nonfinite, gen, quant

pytestmark = pytest.mark.gpu

# (n, c, h, w, oh, ow): widths of every remainder modulo 4, one column, two, a block's last thread partly used, the widest
# row of one block and the first that is too wide, scales of exactly one and just above
SHAPES = [(1, 3, 37, 61, 11, 17), (2, 1, 40, 62, 13, 40), (1, 2, 33, 63, 5, 9), (3, 1, 64, 130, 31, 129),
          (1, 1, 9, 1, 4, 1), (1, 1, 30, 2, 7, 2), (1, 1, 20, 513, 3, 100), (1, 1, 7, 2047, 2, 341),
          (1, 1, 6, 2049, 3, 700), (1, 1, 301, 5, 299, 4), (1, 1, 12, 4095, 4, 1365), (1, 1, 12, 4098, 4, 1365),
          (1, 1, 23, 50, 23, 49), (1, 1, 100, 96, 99, 95)]
HALF_ULP = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def close(got, ref, dtype):
    got = got.detach().cpu().float().numpy().astype(np.float64)
    bar = 1e-6 + 1e-5 * np.abs(ref) + HALF_ULP[dtype] * np.abs(ref) * (1 + 1e-4)
    if dtype == torch.float16:
        bar = bar + 2.0 ** -25
    assert (np.abs(got - ref) <= bar).all(), float((np.abs(got - ref) - bar).max())


def off_by(t, dev, shift):
    """The same values in a buffer whose first element is `shift` elements past an aligned address."""
    flat = torch.empty(t.numel() + shift, dtype=t.dtype, device=dev)
    view = flat[shift:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("filt", ["bicubic", "bilinear"])
@pytest.mark.parametrize("shape", SHAPES)
def test_any_width(ops, oracle, dev, dtype, filt, shape):
    n, c, h, w, oh, ow = shape
    fwd, bwd, ofwd, obwd = {
        "bicubic": (ops.upsample_bicubic2d_aa, ops.upsample_bicubic2d_aa_grad, oracle.bicubic_aa_fwd,
                    oracle.bicubic_aa_bwd),
        "bilinear": (ops.upsample_bilinear2d_aa, ops.upsample_bilinear2d_aa_backward, oracle.bilinear_aa_fwd,
                     oracle.bilinear_aa_bwd)}[filt]
    x, x32 = quant(torch.rand((n, c, h, w), generator=gen(90)), dtype)
    ref = ofwd(x32, (oh, ow), False)
    for shift in (0, 1, 2):
        close(fwd(off_by(x, dev, shift), (oh, ow), False), ref, dtype)
    g, g32 = quant(torch.rand((n, c, oh, ow), generator=gen(91)), dtype)
    ref = obwd(g32, (h, w), False, definition="gather")
    close(bwd(g.to(dev), (oh, ow), (n, c, h, w), False), ref, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
def test_grad_input_at_any_alignment(ops, oracle, dev, dtype):
    g, g32 = quant(torch.rand((1, 2, 9, 21), generator=gen(92)), dtype)
    ref = oracle.bicubic_aa_bwd(g32, (30, 64), False, definition="gather")
    for shift in (0, 1, 2, 3):
        out = off_by(torch.full((1, 2, 30, 64), 7.0, dtype=dtype), dev, shift)
        ops.upsample_bicubic2d_aa_grad(g.to(dev), (9, 21), (1, 2, 30, 64), False, out=out)
        close(out, ref, dtype)


def test_windows_past_the_input_give_zero(ops, oracle, dev):
    x = torch.rand((1, 2, 24, 33), generator=gen(93))
    for size in ((30, 40), (12, 15)):
        y = ops.upsample_bicubic2d_aa(x.to(dev), size, False, scales=(0.25, 0.4))
        close(y, oracle.bicubic_aa_fwd(x.numpy(), size, False, (0.25, 0.4)), torch.float32)
        g = torch.rand((1, 2) + size, generator=gen(97))
        gi = ops.upsample_bicubic2d_aa_grad(g.to(dev), size, (1, 2, 24, 33), False, scales=(0.25, 0.4))
        close(gi, oracle.bicubic_aa_bwd(g.numpy(), (24, 33), False, (0.25, 0.4), definition="gather"), torch.float32)


def test_non_finite_values_at_odd_widths(ops, oracle, dev):
    rng = np.random.default_rng(94)
    x = _poison(torch.rand((1, 2, 41, 57), generator=gen(95)), rng, 6)
    _same_nonfinite(ops.upsample_bicubic2d_aa(x.to(dev), (13, 19), False), oracle.bicubic_aa_fwd(x.numpy(), (13, 19), False),
                    "forward")
    g = _poison(torch.rand((1, 2, 13, 19), generator=gen(96)), rng, 4)
    _same_nonfinite(ops.upsample_bicubic2d_aa_grad(g.to(dev), (13, 19), (1, 2, 41, 57), False),
                    oracle.bicubic_aa_bwd(g.numpy(), (41, 57), False, definition="gather"), "backward")


# one long axis: its tables come from a thread per index (two launches), short ones from a cluster (one)
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("filt", ["bicubic", "bilinear"])
@pytest.mark.parametrize("shape", [(1, 1, 8193, 40, 2731, 20), (1, 1, 20011, 33, 5003, 11), (1, 1, 6, 8193, 3, 4001),
                                   (1, 2, 3, 5000, 5, 9000), (1, 1, 8192, 36, 4096, 18)])
def test_long_axes(ops, oracle, dev, dtype, filt, shape):
    n, c, h, w, oh, ow = shape
    fwd, bwd, ofwd, obwd = {
        "bicubic": (ops.upsample_bicubic2d_aa, ops.upsample_bicubic2d_aa_grad, oracle.bicubic_aa_fwd,
                    oracle.bicubic_aa_bwd),
        "bilinear": (ops.upsample_bilinear2d_aa, ops.upsample_bilinear2d_aa_backward, oracle.bilinear_aa_fwd,
                     oracle.bilinear_aa_bwd)}[filt]
    x, x32 = quant(torch.rand((n, c, h, w), generator=gen(98)), dtype)
    close(fwd(x.to(dev), (oh, ow), False), ofwd(x32, (oh, ow), False), dtype)
    g, g32 = quant(torch.rand((n, c, oh, ow), generator=gen(99)), dtype)
    g = g.to(dev)
    ops.reset_launch_count()
    gi = bwd(g, (oh, ow), (n, c, h, w), False)
    assert ops.launch_count() == (3 if max(shape) > 8192 else 2)
    close(gi, obwd(g32, (h, w), False, definition="gather"), dtype)


# Sizes at which the streaming forward and the band backward take the call (small calls go to a thread per element): every load
# width, a block's last thread partly used, the widest rows, scales just above one
REACHED = [("bicubic", "forward", (1, 2, 33, 63, 5, 9)), ("bicubic", "forward", (1, 2, 40, 62, 8, 12)),
           ("bicubic", "forward", (1, 3, 37, 64, 11, 17)), ("bicubic", "forward", (1, 1, 7, 2047, 2, 341)),
           ("bicubic", "forward", (1, 1, 9, 2048, 3, 400)), ("bicubic", "forward", (64, 1, 100, 96, 99, 95)),
           ("bicubic", "forward", (64, 1, 64, 130, 31, 129)), ("bicubic", "forward", (3, 1, 700, 5, 30, 1)),
           ("bilinear", "forward", (1, 3, 64, 130, 11, 23)), ("bilinear", "forward", (1, 2, 60, 61, 10, 10)),
           ("bilinear", "forward", (2, 2, 36, 64, 6, 12)), ("bilinear", "forward", (1, 1, 40, 2047, 6, 341)),
           ("bilinear", "forward", (256, 1, 100, 96, 99, 95)), ("bicubic", "backward", (1, 2, 33, 63, 5, 9)),
           ("bicubic", "backward", (1, 1, 12, 4095, 4, 1365)), ("bicubic", "backward", (1, 1, 100, 96, 99, 95)),
           ("bilinear", "backward", (64, 1, 100, 96, 99, 95)), ("bilinear", "backward", (64, 1, 20, 513, 3, 100)),
           ("bilinear", "backward", (16, 1, 12, 4095, 4, 1365)), ("bilinear", "backward", (128, 2, 37, 62, 11, 17))]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("filt,way,shape", REACHED)
def test_streaming_and_band_kernels(ops, oracle, dev, dtype, filt, way, shape):
    n, c, h, w, oh, ow = shape
    kernel = f"{filt}_aa_forward_stream" if way == "forward" else f"{filt}_aa_backward_band"
    assert ops.debug_plan(kernel, 4 if dtype == torch.float32 else 2, shape) is not None
    if way == "forward":
        x, x32 = quant(torch.rand((n, c, h, w), generator=gen(100)), dtype)
        ref = getattr(oracle, f"{filt}_aa_fwd")(x32, (oh, ow), False)
        for shift in (0, 1, 2):
            close(getattr(ops, f"upsample_{filt}2d_aa")(off_by(x, dev, shift), (oh, ow), False), ref, dtype)
        return
    bwd = ops.upsample_bicubic2d_aa_grad if filt == "bicubic" else ops.upsample_bilinear2d_aa_backward
    g, g32 = quant(torch.rand((n, c, oh, ow), generator=gen(101)), dtype)
    ref = getattr(oracle, f"{filt}_aa_bwd")(g32, (h, w), False, definition="gather")
    for shift in (0, 1, 3):
        out = off_by(torch.full((n, c, h, w), 7.0, dtype=dtype), dev, shift)
        bwd(g.to(dev), (oh, ow), (n, c, h, w), False, out=out)
        close(out, ref, dtype)
