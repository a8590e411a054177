"""Two-phase aclnn calls over torch CUDA tensors. torch supplies device memory and the current stream only."""
import ctypes

import torch

from . import (ACL_BF16, ACL_DOUBLE, ACL_FLOAT, ACL_FLOAT16, ACL_FORMAT_NCDHW, ACL_FORMAT_NCHW, ACL_FORMAT_NCL, ACL_FORMAT_ND,
               ACL_FORMAT_NDHWC, ACL_FORMAT_NHWC,
               ACL_INT32, ACL_INT64, ACL_OPT_DETERMINISTIC, ACL_UINT8, lib, native_module)

__all__ = [
    "AclnnError", "acl_tensor", "int_array", "bool_array", "float_array", "resize", "two_phase", "set_deterministic", "set_backward_algo",
    "launch_count", "reset_launch_count", "async_copy_timeouts", "last_error", "debug_axis_table", "debug_plan", "upsample_nearest2d",
    "upsample_nearest2d_backward", "upsample_bilinear2d", "upsample_bilinear2d_no_alloc",
    "upsample_bilinear2d_backward", "upsample_bicubic2d", "upsample_bicubic2d_backward", "upsample_bilinear2d_aa",
    "upsample_bilinear2d_aa_backward", "upsample_nearest_exact2d", "upsample_nearest_exact2d_backward",
    "upsample_nearest_exact1d", "upsample_nearest_exact1d_backward", "upsample_nearest3d",
    "upsample_nearest3d_backward", "upsample_trilinear3d", "upsample_trilinear3d_backward", "grid_sampler3d",
    "grid_sampler3d_backward", "upsample_bicubic2d_aa",
    "upsample_bicubic2d_aa_grad", "grid_sampler2d", "grid_sampler2d_backward", "Workspace",
]

_DTYPES = {torch.float32: ACL_FLOAT, torch.float16: ACL_FLOAT16, torch.bfloat16: ACL_BF16, torch.float64: ACL_DOUBLE,
           torch.uint8: ACL_UINT8, torch.int32: ACL_INT32, torch.int64: ACL_INT64}
_FORMATS = {"NCHW": ACL_FORMAT_NCHW, "NHWC": ACL_FORMAT_NHWC, "ND": ACL_FORMAT_ND, "NCL": ACL_FORMAT_NCL,
            "NCDHW": ACL_FORMAT_NCDHW, "NDHWC": ACL_FORMAT_NDHWC}


class AclnnError(RuntimeError):
    def __init__(self, api, status):
        self.status = status
        super().__init__(f"{api} returned {status}: {last_error()}")


_native = None


def native():
    """The native binding (loaded once; OSError if it has not been built)."""
    global _native
    if _native is None:
        module = native_module()
        module.set_classes(AclnnError, Workspace)
        _native = module
    return _native


def last_error():
    return lib().aclGetRecentErrMsg().decode()


class _Handle:
    """Owns one acl object and destroys it with the matching destructor."""

    def __init__(self, ptr, destroy, keep=None):
        self.ptr = ptr
        self._destroy = destroy
        self._keep = keep

    def __del__(self):
        if self.ptr:
            self._destroy(self.ptr)
            self.ptr = None


def acl_tensor(t, fmt="NCHW"):
    """aclTensor view of a torch tensor: its sizes, strides (elements) and data pointer; offset 0."""
    dims = (ctypes.c_int64 * t.dim())(*t.shape)
    strides = (ctypes.c_int64 * t.dim())(*t.stride())
    ptr = lib().aclCreateTensor(dims, t.dim(), _DTYPES[t.dtype], strides, 0, _FORMATS[fmt], dims, t.dim(),
                                ctypes.c_void_p(t.data_ptr()))
    if not ptr:
        raise AclnnError("aclCreateTensor", -1)
    return _Handle(ptr, lib().aclDestroyTensor, keep=t)


def int_array(values):
    arr = (ctypes.c_int64 * len(values))(*values)
    return _Handle(lib().aclCreateIntArray(arr, len(values)), lib().aclDestroyIntArray)


def float_array(values):
    arr = (ctypes.c_float * len(values))(*values)
    return _Handle(lib().aclCreateFloatArray(arr, len(values)), lib().aclDestroyFloatArray)


def bool_array(values):
    arr = (ctypes.c_bool * len(values))(*values)
    return _Handle(lib().aclCreateBoolArray(arr, len(values)), lib().aclDestroyBoolArray)


class Workspace:
    """Grow-only device workspace reused across calls (avoids an allocation per call in timed loops)."""

    def __init__(self, device="cuda"):
        self.device = device
        self.buf = None

    def get(self, nbytes):
        if nbytes == 0:
            return None, 0
        if self.buf is None or self.buf.numel() < nbytes:
            self.buf = torch.empty(nbytes, dtype=torch.uint8, device=self.device)
        return self.buf, nbytes


def two_phase(name, args, device, workspace=None, stream=None):
    """Run `<name>GetWorkspaceSize(*args, &ws, &executor)` then `<name>(workspace, ws, executor, stream)`."""
    L = lib()
    ws_size = ctypes.c_uint64(0)
    executor = ctypes.c_void_p(None)
    status = getattr(L, name + "GetWorkspaceSize")(*args, ctypes.byref(ws_size), ctypes.byref(executor))
    if status != 0:
        raise AclnnError(name + "GetWorkspaceSize", status)
    buf = None
    if ws_size.value > 0:
        if workspace is not None:
            buf, _ = workspace.get(ws_size.value)
        else:
            buf = torch.empty(ws_size.value, dtype=torch.uint8, device=device)
    if stream is None:
        stream = torch.cuda.current_stream(device).cuda_stream
    status = getattr(L, name)(ctypes.c_void_p(buf.data_ptr() if buf is not None else None), ws_size.value, executor,
                              ctypes.c_void_p(stream))
    if status != 0:
        raise AclnnError(name, status)
    return ws_size.value


def set_deterministic(flag):
    lib().aclrtCtxSetSysParamOpt(ACL_OPT_DETERMINISTIC, 1 if flag else 0)


def set_backward_algo(algo):
    status = lib().opscvSetBackwardAlgo({"gather": 0, "atomic": 1}.get(algo, algo))
    if status != 0:
        raise AclnnError("opscvSetBackwardAlgo", status)


def launch_count():
    return lib().opscvGetLaunchCount()


def reset_launch_count():
    lib().opscvResetLaunchCount()


def async_copy_timeouts():
    """Bounded device-side waits that ran out (0 in a healthy run)."""
    return lib().opscvGetAsyncCopyTimeouts()


def debug_axis_table(kind, in_size, out_size, align=False, user_scale=0.0):
    """Index / weight tables as the device builds them, copied to numpy arrays (see opscvDebugAxisTable)."""
    import numpy as np
    L = lib()
    kinds = {"nearest_fwd": 0, "nearest_bwd": 1, "bilinear": 2, "bicubic_aa": 3, "bilinear_aa": 4}
    k = kinds[kind]
    n = in_size if k == 1 else out_size
    i0 = np.zeros(n, dtype=np.int32)
    i1 = np.zeros(n, dtype=np.int32)
    taps = ctypes.c_int32(0)
    f0 = None
    if k == 2:
        f0 = np.zeros(n, dtype=np.float32)
    if k >= 3:
        status = L.opscvDebugAxisTable(k, in_size, out_size, int(align), user_scale, None, None, None,
                                       ctypes.byref(taps))
        if status != 0:
            raise AclnnError("opscvDebugAxisTable", status)
        f0 = np.zeros((n, taps.value), dtype=np.float32)
    status = L.opscvDebugAxisTable(k, in_size, out_size, int(align), user_scale, i0.ctypes.data, i1.ctypes.data,
                                   f0.ctypes.data if f0 is not None else None, ctypes.byref(taps))
    if status != 0:
        raise AclnnError("opscvDebugAxisTable", status)
    return i0, i1, f0


def debug_plan(kind, elem_size, sizes, fmt="NCHW", align=False, scales=(0.0, 0.0)):
    """The launch shape of a kernel for these sizes (see opscvDebugPlan), or None where it does not take the call."""
    taken = ctypes.c_int32(0)
    values = (ctypes.c_int64 * 8)()
    kinds = {"bilinear_backward_walk": 0, "bicubic_backward_walk": 1, "bicubic_aa_forward_stream": 2,
             "bicubic_aa_backward_band": 3, "bilinear_aa_forward_stream": 4, "bilinear_aa_backward_band": 5}
    status = lib().opscvDebugPlan(kinds[kind], elem_size, _FORMATS[fmt], (ctypes.c_int64 * 6)(*sizes), int(align),
                                  (ctypes.c_double * 2)(*scales), ctypes.byref(taken), values)
    if status != 0:
        raise AclnnError("opscvDebugPlan", status)
    return list(values) if taken.value else None


def _out_shape(x, out_hw, fmt):
    if fmt == "NHWC":
        return (x.shape[0], out_hw[0], out_hw[1], x.shape[3])
    return (x.shape[0], x.shape[1], out_hw[0], out_hw[1])


# ---- operators ------------------------------------------------------------------------------------------------
# Each wrapper is one call of the native binding (csrc/py_binding.cpp), which allocates the result unless `out` is given,
# builds the acl objects and runs both phases on the current stream of the tensor's device.

def upsample_nearest2d(x, out_hw, fmt="NCHW", scales=None, out=None, workspace=None):
    return native().upsample_nearest2d(x, out_hw, fmt, scales, out, workspace)


def upsample_nearest2d_backward(grad_out, out_hw, input_size, fmt="NCHW", scales=(0.0, 0.0), out=None,
                                workspace=None):
    return native().upsample_nearest2d_backward(grad_out, out_hw, input_size, fmt, scales, out, workspace)


def upsample_bilinear2d(x, out_hw, align_corners=False, fmt="NCHW", scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_bilinear2d(x, out_hw, align_corners, fmt, scales, out, workspace)


def upsample_bilinear2d_no_alloc(x, out_hw, align_corners=False, fmt="NCHW", scales=(0.0, 0.0), out=None):
    """opscvUpsampleBilinear2dNoAlloc: one call, no workspace (tap tables live in the library's device image)."""
    out = torch.empty(_out_shape(x, out_hw, fmt), dtype=x.dtype, device=x.device) if out is None else out
    assert x.is_contiguous() and out.is_contiguous()
    n, c, h, w = (x.shape[0], x.shape[3], x.shape[1], x.shape[2]) if fmt == "NHWC" else tuple(x.shape)
    with torch.cuda.device(x.device):
        status = lib().opscvUpsampleBilinear2dNoAlloc(
            x.data_ptr(), out.data_ptr(), _DTYPES[x.dtype], _FORMATS[fmt], n, c, h, w, int(out_hw[0]), int(out_hw[1]),
            bool(align_corners), float(scales[0]), float(scales[1]), torch.cuda.current_stream(x.device).cuda_stream)
    if status != 0:
        raise AclnnError("opscvUpsampleBilinear2dNoAlloc", status)
    return out


def upsample_bilinear2d_backward(grad_out, out_hw, input_size, align_corners=False, fmt="NCHW", scales=(0.0, 0.0),
                                 out=None, out_dtype=None, v2=False, workspace=None):
    if out is None and out_dtype is not None:
        out = torch.empty(tuple(input_size), dtype=out_dtype, device=grad_out.device)
    run = native().upsample_bilinear2d_backward_v2 if v2 else native().upsample_bilinear2d_backward
    return run(grad_out, out_hw, input_size, align_corners, fmt, scales, out, workspace)


def upsample_bicubic2d_aa(x, out_hw, align_corners=False, scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_bicubic2d_aa(x, out_hw, align_corners, "NCHW", scales, out, workspace)


def upsample_bicubic2d_aa_grad(grad_out, out_hw, input_size, align_corners=False, scales=(0.0, 0.0), out=None,
                               workspace=None):
    return native().upsample_bicubic2d_aa_grad(grad_out, out_hw, input_size, align_corners, "NCHW", scales, out,
                                               workspace)


def upsample_nearest_exact2d(x, out_hw, fmt="NCHW", scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_nearest_exact2d(x, out_hw, fmt, scales, out, workspace)


def upsample_nearest_exact2d_backward(grad_out, out_hw, input_size, scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_nearest_exact2d_backward(grad_out, out_hw, input_size, "NCHW", scales, out, workspace)


def upsample_nearest_exact1d(x, out_l, scale=0.0, fmt="NCL", out=None, workspace=None):
    return native().upsample_nearest_exact1d(x, out_l, scale, fmt, out, workspace)


def upsample_nearest_exact1d_backward(grad_out, out_l, input_size, scale=0.0, fmt="NCL", out=None, workspace=None):
    return native().upsample_nearest_exact1d_backward(grad_out, out_l, input_size, scale, fmt, out, workspace)


def upsample_nearest3d(x, out_dhw, fmt="NCDHW", scales=(0.0, 0.0, 0.0), exact=False, out=None, workspace=None):
    return native().upsample_nearest3d(x, out_dhw, fmt, scales, exact, out, workspace)


def upsample_nearest3d_backward(grad_out, out_dhw, input_size, fmt="NCDHW", scales=(0.0, 0.0, 0.0), exact=False,
                                out=None, workspace=None):
    return native().upsample_nearest3d_backward(grad_out, out_dhw, input_size, fmt, scales, out, workspace, exact)


def upsample_trilinear3d(x, out_dhw, align_corners=False, fmt="NCDHW", scales=(0.0, 0.0, 0.0), out=None,
                         workspace=None):
    return native().upsample_trilinear3d(x, out_dhw, align_corners, fmt, scales, out, workspace)


def upsample_trilinear3d_backward(grad_out, out_dhw, input_size, align_corners=False, fmt="NCDHW",
                                  scales=(0.0, 0.0, 0.0), out=None, workspace=None):
    """input_size is (N, C, D, H, W) in either format, as in the reference."""
    return native().upsample_trilinear3d_backward(grad_out, out_dhw, input_size, align_corners, fmt, scales, out,
                                                  workspace)


def upsample_bilinear2d_aa(x, out_hw, align_corners=False, scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_bilinear2d_aa(x, out_hw, align_corners, "NCHW", scales, out, workspace)


def upsample_bilinear2d_aa_backward(grad_out, out_hw, input_size, align_corners=False, scales=(0.0, 0.0), out=None,
                                    workspace=None):
    return native().upsample_bilinear2d_aa_backward(grad_out, out_hw, input_size, align_corners, "NCHW", scales, out,
                                                    workspace)


def upsample_bicubic2d(x, out_hw, align_corners=False, fmt="NCHW", scales=(0.0, 0.0), out=None, workspace=None):
    return native().upsample_bicubic2d(x, out_hw, align_corners, fmt, scales, out, workspace)


def upsample_bicubic2d_backward(grad_out, out_hw, input_size, align_corners=False, fmt="NCHW", scales=(0.0, 0.0),
                                out=None, workspace=None):
    return native().upsample_bicubic2d_backward(grad_out, out_hw, input_size, align_corners, fmt, scales, out, workspace)


def resize(x, scales, mode="bilinear", fmt="NCHW", out=None, workspace=None):
    """aclnnResize: `scales` has one factor per dimension of x; the output extent is floor(extent * factor)."""
    if out is None:
        h_dim, w_dim = (1, 2) if fmt == "NHWC" else (2, 3)
        out_hw = (int(x.shape[h_dim] * float(scales[h_dim])), int(x.shape[w_dim] * float(scales[w_dim])))
        out = torch.empty(_out_shape(x, out_hw, fmt), dtype=x.dtype, device=x.device)
    tx, ty, sc = acl_tensor(x, fmt), acl_tensor(out, fmt), float_array([float(v) for v in scales])
    two_phase("aclnnResize", [tx.ptr, sc.ptr, mode.encode(), ty.ptr], x.device, workspace)
    return out


def grid_sampler2d(x, grid, interpolation=0, padding=0, align_corners=False, out=None, workspace=None):
    return native().grid_sampler(x, grid, int(interpolation), int(padding), align_corners, None, out, workspace)


def grid_sampler2d_backward(grad_out, x, grid, interpolation=0, padding=0, align_corners=False, mask=(True, True),
                            input_grad=None, grid_grad=None, workspace=None):
    return native().grid_sampler_backward(grad_out, x, grid, int(interpolation), int(padding), align_corners, mask, None,
                                          input_grad, grid_grad, workspace)


def grid_sampler3d(x, grid, interpolation=0, padding=0, align_corners=False, fmt="NCDHW", out=None, workspace=None):
    return native().grid_sampler(x, grid, int(interpolation), int(padding), align_corners, fmt, out, workspace)


def grid_sampler3d_backward(grad_out, x, grid, interpolation=0, padding=0, align_corners=False, mask=(True, True),
                            fmt="NCDHW", input_grad=None, grid_grad=None, workspace=None):
    return native().grid_sampler_backward(grad_out, x, grid, int(interpolation), int(padding), align_corners, mask, fmt,
                                          input_grad, grid_grad, workspace)
