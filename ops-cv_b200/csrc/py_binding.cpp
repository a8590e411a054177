// The Python caller's fast path: one native call per operator. It reads the tensors' metadata directly, builds the acl
// objects on the stack and runs both phases of the aclnn call on the current stream. The same steps made from Python
// through ctypes (an aclTensor per tensor, an aclIntArray per size, two calls with by-reference results) cost 20 to 35 us
// a call, several times the GPU time of a small one; this costs about 3 us.
//
// The functions take positional arguments in the order of the wrappers in aclnn.py, which document them.
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/Functions.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>

#include <string>

#include "host_common.h"

namespace {

PyObject* g_error = nullptr; // AclnnError(api, status)
PyObject* g_workspace = nullptr; // aclnn.Workspace
PyObject* g_bufName = nullptr;

// Thrown after a Python exception has been set.
struct Raised {};

[[noreturn]] void Raise(PyObject* type, const char* text)
{
    PyErr_SetString(type, text);
    throw Raised{};
}

const at::Tensor& TensorOf(PyObject* o)
{
    if (!THPVariable_Check(o)) {
        Raise(PyExc_TypeError, "expected a torch.Tensor");
    }
    return THPVariable_Unpack(o);
}
int64_t IntOf(PyObject* o)
{
    PyObject* index = PyNumber_Index(o);
    if (index == nullptr) {
        throw Raised{};
    }
    const long long v = PyLong_AsLongLong(index);
    Py_DECREF(index);
    if (v == -1 && PyErr_Occurred()) {
        throw Raised{};
    }
    return v;
}
double DoubleOf(PyObject* o) // float(o)
{
    if (PyFloat_CheckExact(o)) {
        return PyFloat_AS_DOUBLE(o);
    }
    PyObject* f = PyNumber_Float(o);
    if (f == nullptr) {
        throw Raised{};
    }
    const double v = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return v;
}
bool BoolOf(PyObject* o)
{
    const int v = PyObject_IsTrue(o);
    if (v < 0) {
        throw Raised{};
    }
    return v != 0;
}

// A Python sequence's items (a tuple or list as it is, anything else through a temporary).
class Items {
public:
    explicit Items(PyObject* o) : seq_(PySequence_Fast(o, "expected a sequence"))
    {
        if (seq_ == nullptr) {
            throw Raised{};
        }
    }
    ~Items() { Py_DECREF(seq_); }
    Items(const Items&) = delete;
    Items& operator=(const Items&) = delete;
    Py_ssize_t Size() const { return PySequence_Fast_GET_SIZE(seq_); }
    PyObject* operator[](Py_ssize_t i) const
    {
        if (i >= Size()) {
            Raise(PyExc_IndexError, "sequence index out of range");
        }
        return PySequence_Fast_GET_ITEM(seq_, i);
    }

private:
    PyObject* seq_;
};
aclIntArray IntArrayOf(PyObject* o)
{
    const Items items(o);
    aclIntArray a;
    a.v.resize(static_cast<size_t>(items.Size()));
    for (Py_ssize_t i = 0; i < items.Size(); ++i) {
        a.v[i] = IntOf(items[i]);
    }
    return a;
}
struct Scales {
    double v[3];
};
Scales ScalesOf(PyObject* o, int n)
{
    const Items items(o);
    Scales s{};
    for (int i = 0; i < n; ++i) {
        s.v[i] = DoubleOf(items[i]);
    }
    return s;
}

aclFormat FormatOf(PyObject* o)
{
    const char* s = PyUnicode_Check(o) ? PyUnicode_AsUTF8(o) : nullptr;
    const std::string f = s != nullptr ? s : "";
    if (f == "NCHW") { return ACL_FORMAT_NCHW; }
    if (f == "NHWC") { return ACL_FORMAT_NHWC; }
    if (f == "NCDHW") { return ACL_FORMAT_NCDHW; }
    if (f == "NDHWC") { return ACL_FORMAT_NDHWC; }
    if (f == "ND") { return ACL_FORMAT_ND; }
    if (f == "NCL") { return ACL_FORMAT_NCL; }
    PyErr_SetObject(PyExc_KeyError, o);
    throw Raised{};
}
aclDataType DtypeOf(const at::Tensor& t)
{
    switch (t.scalar_type()) {
        case at::kFloat: return ACL_FLOAT;
        case at::kHalf: return ACL_FLOAT16;
        case at::kBFloat16: return ACL_BF16;
        case at::kDouble: return ACL_DOUBLE;
        case at::kByte: return ACL_UINT8;
        case at::kInt: return ACL_INT32;
        case at::kLong: return ACL_INT64;
        default: Raise(PyExc_KeyError, "dtype has no acl counterpart");
    }
}

[[noreturn]] void RaiseStatus(const std::string& api, aclnnStatus status)
{
    PyObject* e = PyObject_CallFunction(g_error, "si", api.c_str(), static_cast<int>(status));
    if (e != nullptr) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    }
    throw Raised{};
}

// An aclTensor on the stack: sizes, strides (elements) and data pointer of a torch tensor.
aclTensor AclOf(const at::Tensor& t, aclFormat format)
{
    aclTensor a;
    if (t.dim() > 8) {
        RaiseStatus("aclCreateTensor", -1);
    }
    a.dims.assign(t.sizes().begin(), t.sizes().end());
    a.strides.assign(t.strides().begin(), t.strides().end());
    a.dtype = DtypeOf(t);
    a.format = format;
    a.data = t.data_ptr();
    return a;
}

struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

// The caller's workspace for `size` bytes: the buffer of an aclnn.Workspace as it is where it is large enough, else the first
// item of what `get(size)` of any object returns: a tensor, another object with data_ptr(), or None. *keep owns it.
struct Held {
    PyObject* o = nullptr;
    ~Held() { Py_XDECREF(o); }
};
void* CallersBuffer(PyObject* workspace, uint64_t size, Held* keep)
{
    if (reinterpret_cast<PyObject*>(Py_TYPE(workspace)) == g_workspace) {
        keep->o = PyObject_GetAttr(workspace, g_bufName);
        if (keep->o == nullptr) {
            throw Raised{};
        }
        if (THPVariable_Check(keep->o) && static_cast<uint64_t>(THPVariable_Unpack(keep->o).numel()) >= size) {
            return THPVariable_Unpack(keep->o).data_ptr();
        }
        Py_CLEAR(keep->o);
    }
    PyObject* got = PyObject_CallMethod(workspace, "get", "K", static_cast<unsigned long long>(size));
    if (got == nullptr) {
        throw Raised{};
    }
    keep->o = PySequence_GetItem(got, 0);
    Py_DECREF(got);
    if (keep->o == nullptr) {
        throw Raised{};
    }
    if (keep->o == Py_None) {
        return nullptr;
    }
    if (THPVariable_Check(keep->o)) {
        return THPVariable_Unpack(keep->o).data_ptr();
    }
    PyObject* at = PyObject_CallMethod(keep->o, "data_ptr", nullptr);
    if (at == nullptr) {
        throw Raised{};
    }
    void* p = PyLong_AsVoidPtr(at);
    Py_DECREF(at);
    if (p == nullptr && PyErr_Occurred()) {
        throw Raised{};
    }
    return p;
}

// Both phases: `first` runs the first phase, `second` is the entry point of the second. The workspace is the caller's or a
// fresh allocation.
template <typename First>
void TwoPhase(const char* name, First first, decltype(&aclnnUpsampleNearest2d) second, const at::Device& device,
              PyObject* workspace)
{
    uint64_t size = 0;
    aclOpExecutor* executor = nullptr;
    aclnnStatus status;
    {
        NoGil nogil;
        status = first(&size, &executor);
    }
    if (status != ACLNN_SUCCESS) {
        RaiseStatus(std::string(name) + "GetWorkspaceSize", status);
    }
    at::Tensor fresh;
    Held held;
    void* buffer = nullptr;
    try {
        if (size > 0 && workspace != Py_None) {
            buffer = CallersBuffer(workspace, size, &held);
        } else if (size > 0) {
            fresh = at::empty({static_cast<int64_t>(size)}, at::TensorOptions().dtype(at::kByte).device(device));
            buffer = fresh.data_ptr();
        }
        if (!device.is_cuda()) {
            Raise(PyExc_ValueError, "expected a cuda device");
        }
    } catch (...) {
        aclDestroyAclOpExecutor(executor);
        throw;
    }
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    {
        NoGil nogil;
        status = second(buffer, size, executor, stream);
    }
    if (status != ACLNN_SUCCESS) {
        RaiseStatus(name, status);
    }
}

PyObject* Give(const at::Tensor& t) { return THPVariable_Wrap(t); }

at::Tensor OutOr(PyObject* out, const at::Tensor& like, std::initializer_list<int64_t> shape)
{
    return out != Py_None ? TensorOf(out) : at::empty(at::IntArrayRef(shape.begin(), shape.size()), like.options());
}
at::Tensor OutOr(PyObject* out, const at::Tensor& like, const aclIntArray& shape)
{
    return out != Py_None ? TensorOf(out) : at::empty(at::IntArrayRef(shape.v.data(), shape.v.size()), like.options());
}
int64_t At(const aclIntArray& a, size_t i)
{
    if (i >= a.v.size()) {
        Raise(PyExc_IndexError, "sequence index out of range");
    }
    return a.v[i];
}
int64_t DimOf(const at::Tensor& t, int64_t i)
{
    if (i >= t.dim()) {
        Raise(PyExc_IndexError, "tuple index out of range");
    }
    return t.size(i);
}
at::Tensor Out2d(PyObject* out, const at::Tensor& x, const aclIntArray& hw, bool last)
{
    if (out != Py_None) {
        return TensorOf(out);
    }
    return last ? OutOr(out, x, {DimOf(x, 0), At(hw, 0), At(hw, 1), DimOf(x, 3)})
                : OutOr(out, x, {DimOf(x, 0), DimOf(x, 1), At(hw, 0), At(hw, 1)});
}
at::Tensor Out3d(PyObject* out, const at::Tensor& x, const aclIntArray& s, bool last)
{
    if (out != Py_None) {
        return TensorOf(out);
    }
    return last ? OutOr(out, x, {DimOf(x, 0), At(s, 0), At(s, 1), At(s, 2), DimOf(x, 4)})
                : OutOr(out, x, {DimOf(x, 0), DimOf(x, 1), At(s, 0), At(s, 1), At(s, 2)});
}

} // namespace

namespace {

using Args = PyObject* const*;

// (x, out_hw, fmt, scales or None, out, workspace)
PyObject* Nearest2d(Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]);
    const aclFormat f = FormatOf(a[2]);
    const at::Tensor y = Out2d(a[4], x, size, f == ACL_FORMAT_NHWC);
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    if (a[3] == Py_None) {
        TwoPhase("aclnnUpsampleNearest2d", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearest2dGetWorkspaceSize(&tx, &size, &ty, n, e);
        }, aclnnUpsampleNearest2d, x.device(), a[5]);
    } else {
        const Scales s = ScalesOf(a[3], 2);
        TwoPhase("aclnnUpsampleNearest2dV2", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearest2dV2GetWorkspaceSize(&tx, &size, static_cast<float>(s.v[0]),
                                                            static_cast<float>(s.v[1]), &ty, n, e);
        }, aclnnUpsampleNearest2dV2, x.device(), a[5]);
    }
    return Give(y);
}

// (x, out_hw, fmt, scales, out, workspace)
PyObject* NearestExact2d(Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]);
    const aclFormat f = FormatOf(a[2]);
    const Scales s = ScalesOf(a[3], 2);
    const at::Tensor y = Out2d(a[4], x, size, f == ACL_FORMAT_NHWC);
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase("aclnnUpsampleNearestExact2d", [&](uint64_t* n, aclOpExecutor** e) {
        return aclnnUpsampleNearestExact2dGetWorkspaceSize(&tx, &size, s.v[0], s.v[1], &ty, n, e);
    }, aclnnUpsampleNearestExact2d, x.device(), a[5]);
    return Give(y);
}

// (x, out_l, scale, fmt, out, workspace)
PyObject* NearestExact1d(Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    aclIntArray size;
    size.v = {IntOf(a[1])};
    const double scale = DoubleOf(a[2]);
    const aclFormat f = FormatOf(a[3]);
    const at::Tensor y = a[4] != Py_None ? TensorOf(a[4]) : OutOr(a[4], x, {DimOf(x, 0), DimOf(x, 1), size.v[0]});
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase("aclnnUpsampleNearestExact1d", [&](uint64_t* n, aclOpExecutor** e) {
        return aclnnUpsampleNearestExact1dGetWorkspaceSize(&tx, &size, scale, &ty, n, e);
    }, aclnnUpsampleNearestExact1d, x.device(), a[5]);
    return Give(y);
}

// (grad_out, out_l, input_size, scale, fmt, out, workspace)
PyObject* NearestExact1dBackward(Args a)
{
    const at::Tensor& g = TensorOf(a[0]);
    aclIntArray size;
    size.v = {IntOf(a[1])};
    const aclIntArray in = IntArrayOf(a[2]);
    const double scale = DoubleOf(a[3]);
    const aclFormat f = FormatOf(a[4]);
    const at::Tensor y = OutOr(a[5], g, in);
    const aclTensor tg = AclOf(g, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase("aclnnUpsampleNearestExact1dBackward", [&](uint64_t* n, aclOpExecutor** e) {
        return aclnnUpsampleNearestExact1dBackwardGetWorkspaceSize(&tg, &size, &in, scale, &ty, n, e);
    }, aclnnUpsampleNearestExact1dBackward, g.device(), a[6]);
    return Give(y);
}

// (grad_out, out_hw, input_size, fmt, scales, out, workspace)
template <typename First>
PyObject* NearestBackward(const char* name, First first, decltype(&aclnnUpsampleNearest2d) second, int axes, Args a)
{
    const at::Tensor& g = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]), in = IntArrayOf(a[2]);
    const aclFormat f = FormatOf(a[3]);
    const Scales s = ScalesOf(a[4], axes);
    const at::Tensor y = OutOr(a[5], g, in);
    const aclTensor tg = AclOf(g, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase(name, [&](uint64_t* n, aclOpExecutor** e) { return first(&tg, &size, &in, s, &ty, n, e); }, second,
             g.device(), a[6]);
    return Give(y);
}
PyObject* Nearest2dBackward(Args a)
{
    return NearestBackward("aclnnUpsampleNearest2dBackward",
        [](auto* g, auto* size, auto* in, const Scales& s, auto* y, uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearest2dBackwardGetWorkspaceSize(g, size, in, s.v[0], s.v[1], y, n, e);
        }, aclnnUpsampleNearest2dBackward, 2, a);
}
PyObject* NearestExact2dBackward(Args a)
{
    return NearestBackward("aclnnUpsampleNearestExact2dBackward",
        [](auto* g, auto* size, auto* in, const Scales& s, auto* y, uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearestExact2dBackwardGetWorkspaceSize(g, size, in, s.v[0], s.v[1], y, n, e);
        }, aclnnUpsampleNearestExact2dBackward, 2, a);
}
PyObject* Nearest3dBackward(Args a) // (..., exact)
{
    if (BoolOf(a[7])) {
        return NearestBackward("aclnnUpsampleNearestExact3dBackward",
            [](auto* g, auto* size, auto* in, const Scales& s, auto* y, uint64_t* n, aclOpExecutor** e) {
                return aclnnUpsampleNearestExact3dBackwardGetWorkspaceSize(g, size, in, s.v[0], s.v[1], s.v[2], y, n, e);
            }, aclnnUpsampleNearestExact3dBackward, 3, a);
    }
    return NearestBackward("aclnnUpsampleNearest3dBackward",
        [](auto* g, auto* size, auto* in, const Scales& s, auto* y, uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearest3dBackwardGetWorkspaceSize(g, size, in, s.v[0], s.v[1], s.v[2], y, n, e);
        }, aclnnUpsampleNearest3dBackward, 3, a);
}

// The four 2-D interpolations: (x, out_hw, align_corners, fmt, scales, out, workspace)
template <typename First>
PyObject* Interp2d(const char* name, First first, decltype(&aclnnUpsampleNearest2d) second, Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]);
    const bool align = BoolOf(a[2]);
    const aclFormat f = FormatOf(a[3]);
    const Scales s = ScalesOf(a[4], 2);
    const at::Tensor y = Out2d(a[5], x, size, f == ACL_FORMAT_NHWC);
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase(name, [&](uint64_t* n, aclOpExecutor** e) { return first(&tx, &size, align, s.v[0], s.v[1], &ty, n, e); },
             second, x.device(), a[6]);
    return Give(y);
}
// and their gradients: (grad_out, out_hw, input_size, align_corners, fmt, scales, out, workspace)
template <typename First>
PyObject* Interp2dBackward(const char* name, First first, decltype(&aclnnUpsampleNearest2d) second, Args a)
{
    const at::Tensor& g = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]), in = IntArrayOf(a[2]);
    const bool align = BoolOf(a[3]);
    const aclFormat f = FormatOf(a[4]);
    const Scales s = ScalesOf(a[5], 2);
    const at::Tensor y = OutOr(a[6], g, in);
    const aclTensor tg = AclOf(g, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase(name, [&](uint64_t* n, aclOpExecutor** e) {
        return first(&tg, &size, &in, align, s.v[0], s.v[1], &ty, n, e);
    }, second, g.device(), a[7]);
    return Give(y);
}
#define OPSCV_INTERP(fn, api) \
    PyObject* fn(Args a) { return Interp2d(#api, api##GetWorkspaceSize, api, a); }
#define OPSCV_INTERP_BACKWARD(fn, api) \
    PyObject* fn(Args a) { return Interp2dBackward(#api, api##GetWorkspaceSize, api, a); }
OPSCV_INTERP(Bilinear2d, aclnnUpsampleBilinear2d)
OPSCV_INTERP(Bicubic2d, aclnnUpsampleBicubic2d)
OPSCV_INTERP(Bilinear2dAA, aclnnUpsampleBilinear2dAA)
OPSCV_INTERP(Bicubic2dAA, aclnnUpsampleBicubic2dAA)
OPSCV_INTERP_BACKWARD(Bilinear2dBackward, aclnnUpsampleBilinear2dBackward)
OPSCV_INTERP_BACKWARD(Bilinear2dBackwardV2, aclnnUpsampleBilinear2dBackwardV2)
OPSCV_INTERP_BACKWARD(Bicubic2dBackward, aclnnUpsampleBicubic2dBackward)
OPSCV_INTERP_BACKWARD(Bilinear2dAABackward, aclnnUpsampleBilinear2dAABackward)
OPSCV_INTERP_BACKWARD(Bicubic2dAAGrad, aclnnUpsampleBicubic2dAAGrad)

// (x, out_dhw, fmt, scales, exact, out, workspace)
PyObject* Nearest3d(Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]);
    const aclFormat f = FormatOf(a[2]);
    const Scales s = ScalesOf(a[3], 3);
    const bool exact = BoolOf(a[4]);
    const at::Tensor y = Out3d(a[5], x, size, f == ACL_FORMAT_NDHWC);
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    if (exact) {
        TwoPhase("aclnnUpsampleNearestExact3d", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearestExact3dGetWorkspaceSize(&tx, &size, s.v[0], s.v[1], s.v[2], &ty, n, e);
        }, aclnnUpsampleNearestExact3d, x.device(), a[6]);
    } else {
        TwoPhase("aclnnUpsampleNearest3d", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnUpsampleNearest3dGetWorkspaceSize(&tx, &size, s.v[0], s.v[1], s.v[2], &ty, n, e);
        }, aclnnUpsampleNearest3d, x.device(), a[6]);
    }
    return Give(y);
}

// (x, out_dhw, align_corners, fmt, scales, out, workspace)
PyObject* Trilinear3d(Args a)
{
    const at::Tensor& x = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]);
    const bool align = BoolOf(a[2]);
    const aclFormat f = FormatOf(a[3]);
    const Scales s = ScalesOf(a[4], 3);
    const at::Tensor y = Out3d(a[5], x, size, f == ACL_FORMAT_NDHWC);
    const aclTensor tx = AclOf(x, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase("aclnnUpsampleTrilinear3d", [&](uint64_t* n, aclOpExecutor** e) {
        return aclnnUpsampleTrilinear3dGetWorkspaceSize(&tx, &size, align, s.v[0], s.v[1], s.v[2], &ty, n, e);
    }, aclnnUpsampleTrilinear3d, x.device(), a[6]);
    return Give(y);
}

// (grad_out, out_dhw, input_size (N, C, D, H, W), align_corners, fmt, scales, out, workspace)
PyObject* Trilinear3dBackward(Args a)
{
    const at::Tensor& g = TensorOf(a[0]);
    const aclIntArray size = IntArrayOf(a[1]), in = IntArrayOf(a[2]);
    const bool align = BoolOf(a[3]);
    const aclFormat f = FormatOf(a[4]);
    const Scales s = ScalesOf(a[5], 3);
    at::Tensor y;
    if (a[6] != Py_None) {
        y = TensorOf(a[6]);
    } else {
        if (in.v.size() != 5) {
            Raise(PyExc_ValueError, "input_size must have five values (N, C, D, H, W)");
        }
        const auto& v = in.v;
        y = f == ACL_FORMAT_NDHWC ? OutOr(a[6], g, {v[0], v[2], v[3], v[4], v[1]}) : OutOr(a[6], g, in);
    }
    const aclTensor tg = AclOf(g, f);
    aclTensor ty = AclOf(y, f);
    TwoPhase("aclnnUpsampleTrilinear3dBackward", [&](uint64_t* n, aclOpExecutor** e) {
        return aclnnUpsampleTrilinear3dBackwardGetWorkspaceSize(&tg, &size, &in, align, s.v[0], s.v[1], s.v[2], &ty, n, e);
    }, aclnnUpsampleTrilinear3dBackward, g.device(), a[7]);
    return Give(y);
}

// (x, grid, interpolation, padding, align_corners, fmt, out, workspace); fmt None: the 2-D operator
PyObject* GridSampler(Args a)
{
    const at::Tensor &x = TensorOf(a[0]), &grid = TensorOf(a[1]);
    const int64_t mode = IntOf(a[2]), pad = IntOf(a[3]);
    const bool align = BoolOf(a[4]);
    const bool volume = a[5] != Py_None;
    const aclFormat f = volume ? FormatOf(a[5]) : ACL_FORMAT_NCHW;
    at::Tensor y;
    if (a[6] != Py_None) {
        y = TensorOf(a[6]);
    } else if (!volume) {
        y = OutOr(a[6], x, {DimOf(x, 0), DimOf(x, 1), DimOf(grid, 1), DimOf(grid, 2)});
    } else if (f == ACL_FORMAT_NDHWC) {
        y = OutOr(a[6], x, {DimOf(grid, 0), DimOf(grid, 1), DimOf(grid, 2), DimOf(grid, 3), DimOf(x, 4)});
    } else {
        y = OutOr(a[6], x, {DimOf(grid, 0), DimOf(x, 1), DimOf(grid, 1), DimOf(grid, 2), DimOf(grid, 3)});
    }
    const aclTensor tx = AclOf(x, f), tg = AclOf(grid, ACL_FORMAT_ND);
    aclTensor ty = AclOf(y, f);
    if (volume) {
        TwoPhase("aclnnGridSampler3D", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnGridSampler3DGetWorkspaceSize(&tx, &tg, mode, pad, align, &ty, n, e);
        }, aclnnGridSampler3D, x.device(), a[7]);
    } else {
        TwoPhase("aclnnGridSampler2D", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnGridSampler2DGetWorkspaceSize(&tx, &tg, mode, pad, align, &ty, n, e);
        }, aclnnGridSampler2D, x.device(), a[7]);
    }
    return Give(y);
}

// (grad_out, x, grid, interpolation, padding, align_corners, mask, fmt, input_grad, grid_grad, workspace)
PyObject* GridSamplerBackward(Args a)
{
    const at::Tensor &g = TensorOf(a[0]), &x = TensorOf(a[1]), &grid = TensorOf(a[2]);
    const int64_t mode = IntOf(a[3]), pad = IntOf(a[4]);
    const bool align = BoolOf(a[5]);
    aclBoolArray mask;
    {
        const Items items(a[6]);
        for (Py_ssize_t i = 0; i < items.Size(); ++i) {
            mask.v.push_back(BoolOf(items[i]) ? 1 : 0);
        }
    }
    const bool volume = a[7] != Py_None;
    const aclFormat f = volume ? FormatOf(a[7]) : ACL_FORMAT_NCHW;
    const at::Tensor gx = a[8] != Py_None ? TensorOf(a[8]) : at::empty_like(x);
    const at::Tensor gg = a[9] != Py_None ? TensorOf(a[9]) : at::empty_like(grid);
    const aclTensor tgo = AclOf(g, f), tx = AclOf(x, f), tg = AclOf(grid, ACL_FORMAT_ND);
    aclTensor tgx = AclOf(gx, f), tgg = AclOf(gg, ACL_FORMAT_ND);
    if (volume) {
        TwoPhase("aclnnGridSampler3DBackward", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnGridSampler3DBackwardGetWorkspaceSize(&tgo, &tx, &tg, mode, pad, align, &mask, &tgx, &tgg, n, e);
        }, aclnnGridSampler3DBackward, x.device(), a[10]);
    } else {
        TwoPhase("aclnnGridSampler2DBackward", [&](uint64_t* n, aclOpExecutor** e) {
            return aclnnGridSampler2DBackwardGetWorkspaceSize(&tgo, &tx, &tg, mode, pad, align, &mask, &tgx, &tgg, n, e);
        }, aclnnGridSampler2DBackward, x.device(), a[10]);
    }
    PyObject* pair = PyTuple_New(2);
    if (pair == nullptr) {
        throw Raised{};
    }
    PyTuple_SET_ITEM(pair, 0, Give(gx));
    PyTuple_SET_ITEM(pair, 1, Give(gg));
    return pair;
}

// Argument count, C++ exceptions.
template <PyObject* (*F)(Args), int N>
PyObject* Entry(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
        return nullptr;
    }
    try {
        return F(args);
    } catch (const Raised&) {
        return nullptr;
    } catch (...) { // by torch's own table: a full device is torch.OutOfMemoryError, and so on
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}
#define OPSCV_METHOD(name, fn, count) \
    {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(Entry<fn, count>)), METH_FASTCALL, nullptr}

// (AclnnError, Workspace)
PyObject* SetClasses(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    if (n != 2) {
        PyErr_Format(PyExc_TypeError, "expected 2 arguments, got %zd", n);
        return nullptr;
    }
    Py_INCREF(args[0]);
    Py_INCREF(args[1]);
    Py_XSETREF(g_error, args[0]);
    Py_XSETREF(g_workspace, args[1]);
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"set_classes", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(SetClasses)), METH_FASTCALL, nullptr},
    OPSCV_METHOD("upsample_nearest2d", Nearest2d, 6),
    OPSCV_METHOD("upsample_nearest2d_backward", Nearest2dBackward, 7),
    OPSCV_METHOD("upsample_nearest_exact2d", NearestExact2d, 6),
    OPSCV_METHOD("upsample_nearest_exact2d_backward", NearestExact2dBackward, 7),
    OPSCV_METHOD("upsample_nearest_exact1d", NearestExact1d, 6),
    OPSCV_METHOD("upsample_nearest_exact1d_backward", NearestExact1dBackward, 7),
    OPSCV_METHOD("upsample_bilinear2d", Bilinear2d, 7),
    OPSCV_METHOD("upsample_bilinear2d_backward", Bilinear2dBackward, 8),
    OPSCV_METHOD("upsample_bilinear2d_backward_v2", Bilinear2dBackwardV2, 8),
    OPSCV_METHOD("upsample_bicubic2d", Bicubic2d, 7),
    OPSCV_METHOD("upsample_bicubic2d_backward", Bicubic2dBackward, 8),
    OPSCV_METHOD("upsample_bilinear2d_aa", Bilinear2dAA, 7),
    OPSCV_METHOD("upsample_bilinear2d_aa_backward", Bilinear2dAABackward, 8),
    OPSCV_METHOD("upsample_bicubic2d_aa", Bicubic2dAA, 7),
    OPSCV_METHOD("upsample_bicubic2d_aa_grad", Bicubic2dAAGrad, 8),
    OPSCV_METHOD("upsample_nearest3d", Nearest3d, 7),
    OPSCV_METHOD("upsample_nearest3d_backward", Nearest3dBackward, 8),
    OPSCV_METHOD("upsample_trilinear3d", Trilinear3d, 7),
    OPSCV_METHOD("upsample_trilinear3d_backward", Trilinear3dBackward, 8),
    OPSCV_METHOD("grid_sampler", GridSampler, 8),
    OPSCV_METHOD("grid_sampler_backward", GridSamplerBackward, 11),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_opscv_torch", "Native calls of the aclnn operators on torch tensors.",
                       -1, kMethods, nullptr, nullptr, nullptr, nullptr};

} // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__opscv_torch(void)
{
    g_bufName = PyUnicode_InternFromString("buf");
    return PyModule_Create(&kModule);
}
