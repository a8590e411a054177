"""The bounds that launch shapes are sized by, against a restatement of the kernels' index arithmetic: a block's shared memory
holds what its rows, columns or windows can ask for. Host arithmetic only (opscvDebugPlan), no GPU."""
import ctypes
import random
import time

import numpy as np
import pytest
import torch

F = np.float32


def bilinear_backward_scale(n_in, n_out, align, user):
    if align:
        return F(n_in - 1) / F(n_out - 1) if n_out > 1 else F(0)
    return F(1) / F(user) if user > 0 else F(n_in) / F(n_out)


def group_starts(n_in, n_out, align, user=0.0):
    """starts[y] = first grads index whose lower tap is y or more, for y = 0 .. n_in (fp32, each operation rounded)."""
    off = F(0) if align else F(0.5)
    scale = bilinear_backward_scale(n_in, n_out, align, user)
    src = (np.arange(n_out, dtype=np.int64).astype(F) + off) * scale - off
    lo = np.minimum(np.floor(np.maximum(src, F(0))).astype(np.int64), n_in - 1)
    return np.searchsorted(lo, np.arange(n_in + 1))


def most(starts, first, count):
    """Most grads indices in the groups first .. first + count - 1, over the given first groups (negative ones are empty)."""
    n_in = len(starts) - 1
    lo = starts[np.clip(first, 0, n_in)]
    hi = starts[np.clip(np.asarray(first) + count, 0, n_in)]
    return int((hi - lo).max())


def check_walk(ops, fmt, elem, n, c, hi, wi, ho, wo, align):
    plan = ops.debug_plan("bilinear_backward_walk", elem, (n, c, hi, wi, ho, wo), fmt, align)
    if plan is None:
        return False
    band, band_cap, group, group_cap, _, _, _, smem = plan
    assert 0 < smem <= (224 if fmt == "NCHW" else 112) * 1024
    rows = group_starts(hi, ho, align)
    assert most(rows, np.arange(0, hi, band) - 1, band + 1) <= band_cap
    if fmt == "NCHW":  # a stage: any run of groups that starts a multiple of them from a band's first
        assert most(rows, np.arange(-1, hi), group) <= group_cap
    else:
        assert most(group_starts(wi, wo, align), np.arange(0, wi, group) - 1, group + 1) <= group_cap
    return True


# long rows and columns: from 2^22 on an index and its half are no longer exact, from 2^24 on indices share a position
LONG = [("NHWC", 4, 4, 1, 11358413, 1, 27879496), ("NHWC", 2, 8, 1, 9000001, 1, 16777216), ("NHWC", 4, 8, 1, 3000001, 1, 8388607),
        ("NHWC", 4, 4, 4000003, 1, 16777215, 2), ("NHWC", 4, 4, 5000000, 1, 20000001, 2), ("NCHW", 4, 1, 5000000, 1, 16777216, 2),
        ("NCHW", 4, 1, 4000001, 2, 33000001, 3), ("NCHW", 2, 1, 8000000, 2, 16777215, 3)]


@pytest.mark.parametrize("fmt,elem,c,hi,wi,ho,wo", LONG)
@pytest.mark.parametrize("align", [False, True])
def test_bilinear_walk_of_long_axes(ops, fmt, elem, c, hi, wi, ho, wo, align):
    taken = check_walk(ops, fmt, elem, 1, c, hi, wi, ho, wo, align)
    if max(ho, wo) > 2 ** 24:
        assert not taken


def test_bilinear_walk_of_random_sizes(ops):
    rng = random.Random(5)
    taken = 0
    for _ in range(1500):
        fmt, elem = rng.choice(["NCHW", "NHWC"]), rng.choice([2, 4])
        hi, wi = int(2 ** rng.uniform(0, 10)), int(2 ** rng.uniform(0, 10))
        ho, wo = int(hi * 2 ** rng.uniform(0, 4)), int(wi * 2 ** rng.uniform(0, 4))
        n, c = rng.randint(1, 20), rng.choice([1, 3, 8, 48, 264])
        taken += check_walk(ops, fmt, elem, n, c, hi, wi, ho, wo, rng.random() < 0.5)
    assert taken > 500


def weight_bits(n_in, n_out, align):
    """Significant bits of the widest weight of an axis, looked up index by index."""
    off = F(0) if align else F(0.5)
    scale = bilinear_backward_scale(n_in, n_out, align, 0.0)
    src = np.maximum((np.arange(n_out).astype(F) + off) * scale - off, F(0))
    delta = src - np.minimum(np.floor(src), F(n_in - 1))
    bits = 0
    for w in np.unique(np.concatenate([delta, F(1) - delta])):
        digits = int(float(w) * 2 ** 60)
        bits = max(bits, digits.bit_length() - (digits & -digits).bit_length() + 1 if digits else 0)
    return bits


def test_weight_bits_of_the_nhwc_walk(ops):
    """Products with weights of few bits are added with one rounding, which is exact only if the bits are not underrated."""
    rng = random.Random(6)
    for k in range(300):
        align = rng.random() < 0.5
        hi, wi = rng.randint(1, 90), rng.randint(1, 90)
        ho, wo = (hi * 2, wi * 4) if k % 3 == 0 else (rng.randint(hi, 4 * hi), rng.randint(wi, 4 * wi))
        plan = ops.debug_plan("bilinear_backward_walk", 2, (1, 8, hi, wi, ho, wo), "NHWC", align)
        if plan is not None:
            assert weight_bits(hi, ho, align) + weight_bits(wi, wo, align) <= plan[6]
    for size, bits in (((1, 8, 64, 64, 128, 128), 4), ((1, 8, 64, 48, 256, 96), 5), ((1, 8, 30, 30, 80, 80), 8)):
        assert ops.debug_plan("bilinear_backward_walk", 2, size, "NHWC")[6] == bits


def test_planning_does_not_grow_with_the_extent(ops):
    """A launch shape is found on the host in every call: microseconds, not one look at every index."""
    best = 1.0
    for _ in range(20):
        start = time.perf_counter()
        ops.debug_plan("bilinear_backward_walk", 2, (1, 8, 4096, 4096, 8192, 8192), "NHWC")
        best = min(best, time.perf_counter() - start)
    assert best < 3e-4


@pytest.mark.parametrize("fmt,c,hi,wi,ho,wo", [("NHWC", 64, 100000, 4, 250000, 9), ("NCHW", 1, 100000, 16, 250000, 40),
                                               ("NHWC", 48, 16000, 16, 32000, 32)])
def test_bilinear_walk_of_one_tall_plane_fills_the_device(ops, fmt, c, hi, wi, ho, wo):
    plan = ops.debug_plan("bilinear_backward_walk", 4, (1, c, hi, wi, ho, wo), fmt)
    assert plan is not None and -(-hi // plan[0]) >= 148  # bands; B200 has 148 SMs
    assert check_walk(ops, fmt, 4, 1, c, hi, wi, ho, wo, False)


def bicubic_rows(n_in, n_out, align, user):
    """First and one past the last grads row of the walk of every grad_input row."""
    off = F(0) if align else F(0.5)
    if align and n_in > 1 and n_out > 1:
        scale, inv = F(n_in - 1) / F(n_out - 1), F(n_out - 1) / F(n_in - 1)
    elif not align and user > 0:
        scale, inv = F(1) / F(user), F(user)
    else:
        scale, inv = F(n_in) / F(n_out), F(n_out) / F(n_in)
    y = np.arange(n_in).astype(F)
    start = np.ceil((y - F(2) + off) * inv - off)
    start = np.clip(start.astype(np.float64), 0, n_out).astype(np.int64)
    h = np.arange(n_out).astype(F)
    src = h * scale if align else (h + off) * scale - off
    end = np.searchsorted(src, y + F(2))
    end[0] = np.searchsorted(np.floor(src), 1, side="right")
    end[-1] = n_out
    return start, np.maximum(end, start)


def check_bicubic(ops, elem, n, c, hi, wi, ho, wo, align, user=0.0, fmt="NCHW"):
    plan = ops.debug_plan("bicubic_backward_walk", elem, (n, c, hi, wi, ho, wo), fmt, align, (user, user))
    if plan is None:
        return False
    band, most_rows, most_open, smem = plan[0], plan[1], plan[2], plan[7]
    assert 0 < smem <= 48 * 1024
    start, end = bicubic_rows(hi, ho, align, user)
    for y0 in range(0, hi, band):
        y1 = min(y0 + band, hi)
        assert end[y0:y1].max() - start[y0:y1].min() <= most_rows
    if hi > 2:  # interior rows whose walks include a grads row
        diff = np.zeros(ho + 1, np.int64)
        np.add.at(diff, start[1:-1], 1)
        np.add.at(diff, end[1:-1], -1)
        assert np.cumsum(diff).max() <= most_open
    return True


@pytest.mark.parametrize("hi,ho", [(60000, 1), (60000, 2), (100000, 2), (20000, 100), (40000, 160000), (200000, 200000),
                                   (1 << 20, 1 << 20), (1 << 20, 1 << 22), ((1 << 20) - 1, 3000001)])
@pytest.mark.parametrize("align", [False, True])
def test_bicubic_walk_of_tall_planes(ops, hi, ho, align):
    taken = check_bicubic(ops, 4, 1, 3, hi, 8, ho, 9, align)
    if not align:
        assert taken


def test_bicubic_walk_of_random_sizes(ops):
    rng = random.Random(8)
    taken = 0
    for _ in range(600):
        hi, wi = int(2 ** rng.uniform(1, 12)), int(2 ** rng.uniform(1, 8))
        ho, wo = max(1, int(hi * 2 ** rng.uniform(-8, 4))), max(1, int(wi * 2 ** rng.uniform(-3, 2)))
        user = rng.choice([0.0, 0.0, ho / hi * rng.uniform(0.97, 1.03)])
        taken += check_bicubic(ops, rng.choice([2, 4]), rng.randint(1, 3), rng.choice([1, 3, 8]), hi, wi, ho, wo,
                               rng.random() < 0.4, user, rng.choice(["NCHW", "NHWC"]))
    assert taken > 200


def aa_windows(n_in, n_out, cubic, align):
    """Per output index: first input index of its window and one past the last."""
    scale = (F(n_in - 1) / F(n_out - 1) if n_out > 1 else F(0)) if align else F(n_in) / F(n_out)
    support = (F(2) if cubic else F(1)) * max(scale, F(1))
    centre = scale * (np.arange(n_out).astype(F) + F(0.5))
    lo = np.maximum(np.floor((centre - support) + F(0.5)).astype(np.int64), 0)
    hi = np.minimum(np.floor((centre + support) + F(0.5)).astype(np.int64), n_in)
    return lo, np.maximum(hi, lo)


def covering(lo, hi, n_in, span):
    """Most windows that reach `span` adjacent input indices, over all places."""
    y = np.arange(n_in)
    start, end = np.searchsorted(hi, y, side="right"), np.searchsorted(lo, y, side="right")
    last = np.minimum(y + span - 1, n_in - 1)
    return int((end[last] - start).max())


def check_aa(ops, cubic, n, c, hi, wi, ho, wo, align):
    name = "bicubic" if cubic else "bilinear"
    lo, top = aa_windows(hi, ho, cubic, align)
    forward = ops.debug_plan(name + "_aa_forward_stream", 4, (n, c, hi, wi, ho, wo), "NCHW", align)
    if forward is not None:
        band, rows, slots = forward[:3]
        assert covering(lo, top, hi, 1) <= slots
        first = np.arange(0, ho, band)
        assert int((top[np.minimum(first + band, ho) - 1] - lo[first]).max()) <= rows
    backward = ops.debug_plan(name + "_aa_backward_band", 4, (n, c, hi, wi, ho, wo), "NCHW", align)
    if backward is not None:
        band, rows, row_slots, col_slots = backward[:4]
        assert covering(lo, top, hi, 4) <= row_slots
        assert covering(lo, top, hi, band) <= rows
        assert covering(*aa_windows(wi, wo, cubic, align), wi, 4) <= col_slots
        assert covering(*aa_windows(wi, wo, cubic, align), wi, 1) <= 5
    return forward is not None, backward is not None


@pytest.mark.parametrize("cubic", [True, False])
@pytest.mark.parametrize("hi,ho", [(1 << 22, 1 << 22), ((1 << 22) - 3, 4100001), (4000000, 1300000), (1 << 23, 8388605),
                                   (16700001, 16690007), ((1 << 24) - 1, 9000001), (25000000, 20000000)])
def test_aa_kernels_of_long_axes(ops, cubic, hi, ho):
    """Past 2^23 rows centres round by so much that an input row can feed more outputs than the kernels keep open."""
    for align in (False, True):
        check_aa(ops, cubic, 1, 1, hi, 8, ho, 2, align)


def test_aa_kernels_of_random_sizes(ops):
    rng = random.Random(9)
    for _ in range(400):
        hi, wi = int(2 ** rng.uniform(0, 12)), int(2 ** rng.uniform(0, 12))
        s = 2 ** rng.uniform(0, 4)
        check_aa(ops, rng.random() < 0.5, rng.randint(1, 64), rng.choice([1, 3, 8]), hi, wi, max(1, int(hi / s)),
                 max(1, int(wi / (s * rng.uniform(0.9, 1.1)))), rng.random() < 0.3)


def test_aa_stream_takes_bands_that_fit(ops):
    """The band that the model of the walk likes best may need more shared memory than there is: another one is taken."""
    assert ops.debug_plan("bilinear_aa_forward_stream", 4, (33, 8, 2397, 1331, 508, 282)) is not None
    wide = ops.debug_plan("bicubic_aa_forward_stream", 4, (62, 3, 2110, 1864, 875, 773))
    assert wide is not None and wide[4] == 1  # and the horizontal weights stay in shared memory


def workspace_size(ops, name, *args):
    ws, ex = ctypes.c_uint64(0), ctypes.c_void_p(None)
    status = getattr(ops.lib(), name + "GetWorkspaceSize")(*args, ctypes.byref(ws), ctypes.byref(ex))
    assert status == 0
    assert ops.lib().aclDestroyAclOpExecutor(ex) == 0
    return ws.value


@pytest.mark.parametrize("shape,stages", [((2, 8, 8, 28, 28, 16, 56, 56), 1), ((1, 2, 4, 3, 5, 4, 200, 5), 2),
                                          ((1, 2, 4, 4, 4, 4, 8, 50), 2)])
def test_trilinear_backward_asks_for_the_scratch_that_it_uses(ops, shape, stages):
    """By planes only the sums of the H stage go through memory; with longer lists of taps those of the W stage as well."""
    n, c, di, hi, wi, do, ho, wo = shape
    grad, gi = torch.zeros((n, c, do, ho, wo), dtype=torch.float16), torch.zeros((n, c, di, hi, wi), dtype=torch.float16)
    tg, ti = ops.acl_tensor(grad, "NCDHW"), ops.acl_tensor(gi, "NCDHW")
    osz, isz = ops.int_array([do, ho, wo]), ops.int_array([n, c, di, hi, wi])
    size = workspace_size(ops, "aclnnUpsampleTrilinear3dBackward", tg.ptr, osz.ptr, isz.ptr, False, 0.0, 0.0, 0.0, ti.ptr)
    w_stage, h_stage = n * c * do * ho * wi * 4, n * c * do * hi * wi * 4
    tables = 20000  # starts, counts and weights of the three axes, every piece rounded up to 256 bytes
    need = h_stage + (w_stage if stages == 2 else 0)
    assert need <= size <= need + tables


@pytest.mark.parametrize("elem,size,walk", [(4, (1, 400, 100, 130, 110, 143), False), (2, (1, 400, 100, 130, 150, 195), False),
                                            (4, (1, 400, 100, 130, 150, 195), True), (4, (1, 400, 100, 130, 200, 261), True),
                                            (4, (1, 25, 100, 130, 110, 143), True), (2, (8, 21, 65, 65, 513, 513), True)])
def test_bilinear_walk_leaves_large_calls_at_small_scales_to_the_tiles(ops, elem, size, walk):
    assert (ops.debug_plan("bilinear_backward_walk", elem, size) is not None) == walk
