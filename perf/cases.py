"""Workloads of the resampling operators, as a user's program calls them: the cases by which the library's speed is judged.

A case is a dict of plain values. Its "op" names what a pass runs:

  bilinear2d   UpsampleBilinear2d, NCHW or NHWC
  pyramid      UpsampleNearest2d (or NearestExact2d) and UpsampleBilinear2d on the same feature map
  image        UpsampleBicubic2dAA or UpsampleBilinear2dAA: anti-aliased down-scaling of images
  bicubic2d    UpsampleBicubic2d
  grid2d       GridSampler2D
  volume       UpsampleNearest3d and UpsampleTrilinear3d on the same volume
  grid3d       GridSampler3D

and "backward" says whether the backward operators run as well. All calls go through the package's two-phase wrappers
on the current stream, with a workspace that the caller keeps; results are allocated by the calls.
"""
import importlib
import math

import torch

ops = importlib.import_module("ops-cv_b200")

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_SIZE = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # one small picture enlarged on its own: launches and host work are all there is
        dict(name="small_picture", op="bilinear2d", dtype="f32", layout="NCHW", n=1, c=3, h=64, w=64, oh=128, ow=128,
             align=False, backward=False),
        # a spatial transformer on small one-channel pictures, a training step: the small end of the grid sampler
        dict(name="small_transformer", op="grid2d", dtype="f32", n=32, c=1, h=28, w=28, oh=28, ow=28, grid="affine",
             padding=0, align=False, deterministic=False, backward=True),
        # the top-down path of a feature pyramid, a training step at 2x in half precision
        dict(name="pyramid", op="pyramid", dtype="f16", n=32, c=256, h=56, w=56, oh=112, ow=112, exact=False,
             backward=True),
        # the logits of a dense-prediction head brought to the size of the picture, corners aligned, odd extents
        dict(name="dense_logits", op="bilinear2d", dtype="f32", layout="NCHW", n=8, c=21, h=65, w=65, oh=513, ow=513,
             align=True, backward=True),
        # channels-last feature maps in bf16, a training step
        dict(name="channels_last", op="bilinear2d", dtype="bf16", layout="NHWC", n=64, c=256, h=64, w=64, oh=128,
             ow=128, align=False, backward=True),
        # photographs brought to the input size of a classifier, with the gradient with respect to the photographs
        dict(name="photos_bicubic", op="image", filter="bicubic", dtype="f32", n=64, c=3, h=1024, w=1024, oh=224,
             ow=224, align=False, backward=True),
        # video frames brought to a ragged smaller size, half precision, no gradient
        dict(name="frames_bilinear", op="image", filter="bilinear", dtype="f16", n=16, c=3, h=720, w=1280, oh=333,
             ow=592, align=False, backward=False),
        # feature maps enlarged by a factor that is no whole number, cubic
        dict(name="bicubic_ragged", op="bicubic2d", dtype="f32", n=8, c=64, h=60, w=80, oh=150, ow=199, align=False,
             backward=True),
        # sampling at random places (ten per cent of them outside), a training step in bf16
        dict(name="grid_random", op="grid2d", dtype="bf16", n=16, c=256, h=64, w=64, oh=128, ow=128, grid="random",
             padding=0, align=False, deterministic=False, backward=True),
        # rotated, scaled and shifted feature maps, a training step that has to be reproducible bit by bit
        dict(name="grid_affine", op="grid2d", dtype="f32", n=32, c=128, h=96, w=96, oh=96, ow=96, grid="affine",
             padding=0, align=False, deterministic=True, backward=True),
        # the decoder of a volumetric network, a training step at 2x in half precision
        dict(name="volume", op="volume", dtype="f16", n=2, c=32, d=32, h=56, w=56, od=64, oh=112, ow=112, align=False,
             backward=True),
        # a volume warped by a deformation field, a training step
        dict(name="volume_warp", op="grid3d", dtype="f32", layout="NCDHW", n=2, c=32, d=32, h=64, w=64, od=32, oh=64,
             ow=64, grid="random", padding=0, align=False, backward=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scaled(rng, extent, lo, hi):
    return max(1, int(round(extent * rng.uniform(lo, hi))))


def _draw_small_picture(rng):
    h, w = _log_int(rng, 16, 160), _log_int(rng, 16, 160)
    s = rng.choice([2.0, rng.uniform(1.2, 4.0)])
    return dict(op="bilinear2d", dtype=rng.choice(["f32", "f16"]), layout="NCHW", n=rng.randint(1, 4),
                c=rng.choice([1, 3, 4]), h=h, w=w, oh=int(h * s), ow=int(w * s), align=rng.random() < 0.25,
                backward=False)


def _draw_small_transformer(rng):
    return dict(op="grid2d", dtype=rng.choice(["f32", "f32", "f16"]), n=_log_int(rng, 1, 64), c=rng.randint(1, 4),
                h=rng.randint(16, 64), w=rng.randint(16, 64), oh=rng.randint(16, 64), ow=rng.randint(16, 64),
                grid="affine", padding=rng.choice([0, 0, 1]), align=rng.random() < 0.5,
                deterministic=rng.random() < 0.3, backward=True)


def _draw_pyramid(rng):
    # a finer level has twice the extent of the coarser one, or one less where its own extent is odd
    h, w = _log_int(rng, 7, 136), _log_int(rng, 7, 168)
    return dict(op="pyramid", dtype=rng.choice(["f16", "bf16", "f32"]), n=_log_int(rng, 1, 32),
                c=32 * rng.randint(2, 16), h=h, w=w, oh=2 * h - rng.choice([0, 0, 1]), ow=2 * w - rng.choice([0, 0, 1]),
                exact=rng.random() < 0.25, backward=True)


def _draw_dense_logits(rng):
    h, w, s = _log_int(rng, 17, 160), _log_int(rng, 17, 160), rng.uniform(2.0, 8.0)
    return dict(op="bilinear2d", dtype=rng.choice(["f32", "f32", "f16", "bf16"]), layout="NCHW", n=_log_int(rng, 1, 16),
                c=_log_int(rng, 1, 150), h=h, w=w, oh=int(h * s), ow=int(w * s), align=rng.random() < 0.6,
                backward=True)


def _draw_channels_last(rng):
    h, w = _log_int(rng, 12, 128), _log_int(rng, 12, 128)
    s = rng.choice([2.0, 2.0, rng.uniform(1.2, 4.0)])
    return dict(op="bilinear2d", dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), layout="NHWC",
                n=_log_int(rng, 1, 64), c=8 * rng.randint(4, 48), h=h, w=w, oh=int(h * s), ow=int(w * s),
                align=rng.random() < 0.25, backward=True)


def _draw_image(rng):
    h, w, s = _log_int(rng, 240, 2048), _log_int(rng, 240, 2048), rng.uniform(1.3, 6.0)
    return dict(op="image", filter=rng.choice(["bicubic", "bilinear"]), dtype=rng.choice(["f32", "f32", "f16", "bf16"]),
                n=_log_int(rng, 1, 64), c=rng.choice([1, 3, 3]), h=h, w=w, oh=int(h / s),
                ow=int(w / (s * rng.uniform(0.9, 1.1))), align=False, backward=rng.random() < 0.5)


def _draw_bicubic(rng):
    h, w = _log_int(rng, 24, 160), _log_int(rng, 24, 160)
    s = rng.choice([2.0, rng.uniform(1.3, 4.0), rng.uniform(1.3, 4.0)])
    return dict(op="bicubic2d", dtype=rng.choice(["f32", "f16", "bf16"]), n=_log_int(rng, 1, 16), c=_log_int(rng, 3, 128),
                h=h, w=w, oh=int(h * s), ow=int(w * s), align=rng.random() < 0.3, backward=rng.random() < 0.7)


def _draw_grid(rng):
    return dict(op="grid2d", dtype=rng.choice(["f32", "bf16", "f16"]), n=_log_int(rng, 1, 32), c=8 * rng.randint(2, 32),
                h=_log_int(rng, 24, 128), w=_log_int(rng, 24, 128), oh=_log_int(rng, 24, 160), ow=_log_int(rng, 24, 160),
                grid=rng.choice(["random", "affine"]), padding=rng.choice([0, 0, 1]), align=rng.random() < 0.3,
                deterministic=rng.random() < 0.4, backward=rng.random() < 0.75)


def _draw_volume(rng):
    d, h, w = _log_int(rng, 8, 48), _log_int(rng, 8, 80), _log_int(rng, 8, 80)
    one = rng.choice([0, 0, 1])
    return dict(op="volume", dtype=rng.choice(["f16", "bf16", "f32"]), n=rng.randint(1, 4), c=8 * rng.randint(1, 16), d=d,
                h=h, w=w, od=2 * d - one, oh=2 * h - one, ow=2 * w - one, align=rng.random() < 0.3, backward=True)


def _draw_volume_warp(rng):
    return dict(op="grid3d", dtype=rng.choice(["f32", "f32", "f16"]), layout=rng.choice(["NCDHW", "NCDHW", "NDHWC"]),
                n=rng.randint(1, 3), c=rng.choice([1, 3, 16, 32, 64]), d=_log_int(rng, 12, 64), h=_log_int(rng, 16, 96),
                w=_log_int(rng, 16, 96), od=_log_int(rng, 12, 64), oh=_log_int(rng, 16, 96), ow=_log_int(rng, 16, 96),
                grid=rng.choice(["random", "affine"]), padding=rng.choice([0, 1]), align=rng.random() < 0.5,
                backward=True)


# the drawing function of each range and the most bytes that a case of it moves
_RANGES = [(_draw_small_picture, 2e6), (_draw_small_transformer, 8e6), (_draw_pyramid, 1.0e9),
           (_draw_dense_logits, 5e8), (_draw_channels_last, 1.0e9), (_draw_image, 1.0e9), (_draw_bicubic, 1.5e8),
           (_draw_grid, 4e8), (_draw_volume, 4e8), (_draw_volume_warp, 1.5e8)]


def draw(rng):
    make, most = rng.choice(_RANGES)
    while True:
        case = make(rng)
        if work(case)["bytes"] <= most:
            return case


def _numel(case):
    """Elements of the input, of the output and of the sampling grid of one operator."""
    k = case["n"] * case["c"]
    if case["op"] in ("volume", "grid3d"):
        point = case["od"] * case["oh"] * case["ow"]
        grid = case["n"] * point * 3 if case["op"] == "grid3d" else 0
        return k * case["d"] * case["h"] * case["w"], k * point, grid
    point = case["oh"] * case["ow"]
    return k * case["h"] * case["w"], k * point, case["n"] * point * 2 if case["op"] == "grid2d" else 0


def work(case):
    """Every tensor that an operator reads or writes once; about the multiplications and additions of its taps."""
    x, y, g = _numel(case)
    taps = {"bilinear2d": 9, "pyramid": 9, "image": 0, "bicubic2d": 35, "grid2d": 8, "volume": 21, "grid3d": 16}[case["op"]]
    forward, flops = x + g + y, taps * y
    if case["op"] == "image":
        flops = 2 * (4 if case["filter"] == "bicubic" else 2) * x
    if case["op"] in ("grid2d", "grid3d"):
        backward, back_flops = (y + x + g) + (x + g), 3 * taps * y
    else:
        backward, back_flops = y + x, flops
    times = 2 if case["op"] in ("pyramid", "volume") else 1
    both = case["backward"]
    return {"bytes": _SIZE[case["dtype"]] * times * (forward + (backward if both else 0)),
            "flops": flops + (back_flops if both else 0)}


def tolerance(case):
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}


def _affine_grid(case, gen):
    """Rotation by up to 30 degrees, scale 0.8 to 1.2, shift by up to a tenth: one transform for each image."""
    n, dims = case["n"], 3 if case["op"] == "grid3d" else 2
    u = torch.rand((n, 5), generator=gen, device="cuda") * 2 - 1
    phi, scale = u[:, 0] * (math.pi / 6), 1 + 0.2 * u[:, 1]
    theta = torch.zeros((n, dims, dims + 1), device="cuda")
    theta[:, 0, 0], theta[:, 0, 1] = scale * torch.cos(phi), -scale * torch.sin(phi)
    theta[:, 1, 0], theta[:, 1, 1] = scale * torch.sin(phi), scale * torch.cos(phi)
    if dims == 3:
        theta[:, 2, 2] = scale
    theta[:, :, dims] = 0.1 * u[:, 2:2 + dims]
    out = (case["od"], case["oh"], case["ow"]) if dims == 3 else (case["oh"], case["ow"])
    return torch.nn.functional.affine_grid(theta, [n, 1, *out], align_corners=case["align"]).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, op = _DTYPES[case["dtype"]], case["op"]
    inner = [case["h"], case["w"]]
    outer = [case["oh"], case["ow"]]
    if op in ("volume", "grid3d"):
        inner, outer = [case["d"]] + inner, [case["od"]] + outer
    last = case.get("layout") in ("NHWC", "NDHWC")
    n, c = case["n"], case["c"]
    shape = [n, *inner, c] if last else [n, c, *inner]
    out_shape = [n, *outer, c] if last else [n, c, *outer]
    state = dict(case=case, size=tuple(outer), shape=tuple(shape), workspace=ops.Workspace())
    if op == "image":
        state["x"] = (torch.randint(0, 256, shape, generator=gen, device="cuda").float() / 255).to(dtype)
    else:
        state["x"] = torch.randn(shape, generator=gen, device="cuda").to(dtype)
    if op in ("grid2d", "grid3d"):
        if case["grid"] == "affine":
            grid = _affine_grid(case, gen)
        else:
            grid = torch.rand([n, *outer, len(outer)], generator=gen, device="cuda") * 2.2 - 1.1
        state["grid"] = grid.to(dtype)
    if case["backward"]:
        state["grad"] = torch.randn(out_shape, generator=gen, device="cuda").to(dtype)
    return state


def _bilinear2d(s):
    case, size, ws = s["case"], s["size"], s["workspace"]
    fmt = case.get("layout", "NCHW")
    align = case.get("align", False)
    out = [ops.upsample_bilinear2d(s["x"], size, align, fmt=fmt, workspace=ws)]
    if case["backward"]:
        out.append(ops.upsample_bilinear2d_backward(s["grad"], size, s["shape"], align, fmt=fmt, workspace=ws))
    return out


def _pyramid(s):
    case, size, ws = s["case"], s["size"], s["workspace"]
    if case["exact"]:
        out = [ops.upsample_nearest_exact2d(s["x"], size, workspace=ws)]
    else:
        out = [ops.upsample_nearest2d(s["x"], size, workspace=ws)]
    if case["backward"]:
        back = ops.upsample_nearest_exact2d_backward if case["exact"] else ops.upsample_nearest2d_backward
        out.append(back(s["grad"], size, s["shape"], workspace=ws))
    return out + _bilinear2d(s)


def _image(s):
    case, size, ws = s["case"], s["size"], s["workspace"]
    if case["filter"] == "bicubic":
        forward, backward = ops.upsample_bicubic2d_aa, ops.upsample_bicubic2d_aa_grad
    else:
        forward, backward = ops.upsample_bilinear2d_aa, ops.upsample_bilinear2d_aa_backward
    out = [forward(s["x"], size, case["align"], workspace=ws)]
    if case["backward"]:
        out.append(backward(s["grad"], size, s["shape"], case["align"], workspace=ws))
    return out


def _bicubic2d(s):
    case, size, ws = s["case"], s["size"], s["workspace"]
    out = [ops.upsample_bicubic2d(s["x"], size, case["align"], workspace=ws)]
    if case["backward"]:
        out.append(ops.upsample_bicubic2d_backward(s["grad"], size, s["shape"], case["align"], workspace=ws))
    return out


def _grid2d(s):
    case, ws = s["case"], s["workspace"]
    out = [ops.grid_sampler2d(s["x"], s["grid"], 0, case["padding"], case["align"], workspace=ws)]
    if case["backward"]:
        if case["deterministic"]:
            ops.set_deterministic(True)
        try:
            out += ops.grid_sampler2d_backward(s["grad"], s["x"], s["grid"], 0, case["padding"], case["align"],
                                               workspace=ws)
        finally:
            if case["deterministic"]:
                ops.set_deterministic(False)
    return out


def _volume(s):
    case, size, ws = s["case"], s["size"], s["workspace"]
    out = [ops.upsample_nearest3d(s["x"], size, workspace=ws),
           ops.upsample_trilinear3d(s["x"], size, case["align"], workspace=ws)]
    if case["backward"]:
        out.append(ops.upsample_nearest3d_backward(s["grad"], size, s["shape"], workspace=ws))
        out.append(ops.upsample_trilinear3d_backward(s["grad"], size, s["shape"], case["align"], workspace=ws))
    return out


def _grid3d(s):
    case, ws = s["case"], s["workspace"]
    fmt = case["layout"]
    out = [ops.grid_sampler3d(s["x"], s["grid"], 0, case["padding"], case["align"], fmt=fmt, workspace=ws)]
    if case["backward"]:
        out += ops.grid_sampler3d_backward(s["grad"], s["x"], s["grid"], 0, case["padding"], case["align"], fmt=fmt,
                                           workspace=ws)
    return out


_RUN = {"bilinear2d": _bilinear2d, "pyramid": _pyramid, "image": _image, "bicubic2d": _bicubic2d, "grid2d": _grid2d,
        "volume": _volume, "grid3d": _grid3d}


def run(state):
    return _RUN[state["case"]["op"]](state)
