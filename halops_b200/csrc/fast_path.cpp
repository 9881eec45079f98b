// Native front of the Python entry points: argument checks, output allocation and the call into the
// C ABI in one CPython call.
//
// A small GEMM runs for 3 to 8 us on the device; the Python wrapper in front of it took the host 8 us
// (quantizer) and 10 us (GEMM), most of it attribute reads of tensors and the conversion of some twenty
// ctypes arguments, so a chain of eager calls ran at the host's pace (128 x 256 x 512 with its
// quantizer: 26 us of host time, 7.4 us of kernels).  Here the same checks read the tensors' fields.
//
// A function below handles the ordinary call: plain CUDA tensors, flags that are real bools, every check
// passed and the C ABI's return code 0.  For anything else it returns None without having
// done anything, and the Python wrapper goes through its own checks, which own all error texts (a call
// that the C ABI refused launches nothing, so it can be made again for its message).

#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "../../include/halops_b200.h"

namespace {

constexpr int kErrLen = 512;

// The signatures are the header's, so a changed one does not compile here until its call is changed too.
using QuantFn = decltype(&hq_group_wise_quant);
using RmsFn = decltype(&hq_rms_norm_quant);
using DenseFn = decltype(&hq_dense_gemm);
using SituFn = decltype(&hq_dense_gemm_situ_quant);
using DescribeGroupFn = decltype(&hq_describe_group_tile);
using MaskedFn = decltype(&hq_group_masked_gemm);
using ContiguousFn = decltype(&hq_group_contiguous_gemm);

// the entry points of the shared library that the Python package has loaded
struct {
    QuantFn quant;
    RmsFn rms;
    DenseFn dense;
    SituFn situ;
    DescribeGroupFn describe_group;
    MaskedFn masked;
    ContiguousFn contiguous;
    decltype(&hq_hold_switches) hold_switches;
} g_fn;

// the package's mode names
int mode_id(PyObject* o) {
    if (!PyUnicode_CheckExact(o)) return -1;
    const char* s = PyUnicode_AsUTF8(o);
    if (s == nullptr) {
        PyErr_Clear();
        return -1;
    }
    if (std::strcmp(s, "w8a8-mxfp8") == 0) return HQ_MODE_W8A8_MXFP8;
    if (std::strcmp(s, "w4a4-mxfp4") == 0) return HQ_MODE_W4A4_MXFP4;
    if (std::strcmp(s, "w4a4-nvfp4") == 0) return HQ_MODE_W4A4_NVFP4;
    if (std::strcmp(s, "w4a8-mxfp4") == 0) return HQ_MODE_W4A8_MXFP4;
    return -1;
}

// A plain strided CUDA tensor (no subclass, no wrapper of a transform) or null.
const at::Tensor* plain_tensor(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage()) return nullptr;
    if (t.unsafeGetTensorImpl()->is_python_dispatch()) return nullptr;
    return &t;
}

bool flag(PyObject* o, int* out) {
    if (o == Py_True || o == Py_False) {
        *out = o == Py_True ? 1 : 0;
        return true;
    }
    return false;
}

bool small_int(PyObject* o, int* out) {  // an int or an IntEnum member
    if (!PyLong_Check(o)) return false;
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(o, &overflow);
    if (overflow != 0 || v < INT32_MIN || v > INT32_MAX) return false;
    *out = int(v);
    return true;
}

bool real(PyObject* o, float* out) {
    if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred() != nullptr) {
        PyErr_Clear();
        return false;
    }
    *out = float(v);
    return true;
}

bool bytes(const at::Tensor& t) { return t.itemsize() == 1; }
bool u8(const at::Tensor& t) { return t.scalar_type() == at::kByte; }

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Gives the interpreter lock away for its lifetime.
class Unlocked {
    PyThreadState* const state_ = PyEval_SaveThread();

public:
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    ~Unlocked() { PyEval_RestoreThread(state_); }
};

// Runs without the interpreter lock, as torch.empty and a ctypes call do: the C ABI call, and the allocation of the
// outputs, which may wait for the device when the allocator has to free memory for it.
template <typename F>
int unlocked(F&& f) {
    char err[kErrLen];
    const Unlocked scope;
    return f(err);
}

// The same for the GEMMs, whose C ABI reads environment switches: they are read before the lock is given away, since an
// assignment to os.environ in another thread moves the array that they are in.
template <typename F>
int unlocked_gemm(F&& f) {
    const struct Held {
        Held() { g_fn.hold_switches(1); }
        Held(const Held&) = delete;
        ~Held() { g_fn.hold_switches(0); }
    } held;
    return unlocked(f);
}

PyObject* pair_of(const at::Tensor& a, const at::Tensor& b) {
    PyObject* const x = THPVariable_Wrap(a);
    PyObject* const y = x != nullptr ? THPVariable_Wrap(b) : nullptr;
    PyObject* const t = y != nullptr ? PyTuple_Pack(2, x, y) : nullptr;
    Py_XDECREF(x);
    Py_XDECREF(y);
    return t;
}

// rows of 16-bit elements as the quantizers read them
bool quant_input(const at::Tensor& x) {
    return x.dim() == 2 && x.stride(1) == 1 && (x.stride(0) * 2) % 16 == 0 &&
           reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
}

// group_wise_quant(input, mode, use_swizzle, use_pdl, output_quant, output_sf)
PyObject* group_wise_quant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    int swizzle, pdl;
    if (nargs != 6 || g_fn.quant == nullptr || at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
    const at::Tensor* const x = plain_tensor(a[0]);
    const int mode = mode_id(a[1]);
    if (x == nullptr || mode < 0 || mode == HQ_MODE_W4A8_MXFP4 || !flag(a[2], &swizzle) || !flag(a[3], &pdl)) Py_RETURN_NONE;
    const bool bf16 = x->scalar_type() == at::kBFloat16;
    if ((!bf16 && x->scalar_type() != at::kHalf) || !quant_input(*x)) Py_RETURN_NONE;
    const int64_t m = x->size(0), k = x->size(1), group = mode == HQ_MODE_W4A4_NVFP4 ? 16 : 32, kb = k / group;
    if (m == 0 || k == 0 || k % group != 0 || (swizzle != 0 && kb % 4 != 0)) Py_RETURN_NONE;
    const int64_t m_sf = swizzle != 0 ? (m + 127) / 128 * 128 : m;
    const int64_t qk = mode == HQ_MODE_W8A8_MXFP8 ? k : k / 2;
    const auto qt = mode == HQ_MODE_W8A8_MXFP8 ? at::kFloat8_e4m3fn : at::kByte;
    at::Tensor q, sf;
    if (a[4] != Py_None) {
        const at::Tensor* const t = plain_tensor(a[4]);
        if (t == nullptr || !t->is_contiguous() || t->scalar_type() != qt || t->numel() != m * qk || t->device() != x->device()) {
            Py_RETURN_NONE;
        }
        q = *t;
    }
    if (a[5] != Py_None) {
        const at::Tensor* const t = plain_tensor(a[5]);
        if (t == nullptr || !t->is_contiguous() || !u8(*t) || t->numel() != m_sf * kb || t->device() != x->device()) {
            Py_RETURN_NONE;
        }
        sf = *t;
    }
    const void* const px = x->data_ptr();
    const int64_t ld = x->stride(0);
    const int dev = x->get_device();
    void* const st = stream_of(*x);
    const auto on_device = at::TensorOptions().device(x->device());
    if (unlocked([&](char* err) {
            if (!q.defined()) q = at::empty({m, qk}, on_device.dtype(qt));
            if (!sf.defined()) sf = at::empty({m_sf, kb}, on_device.dtype(at::kByte));
            return g_fn.quant(px, ld, bf16 ? HQ_DTYPE_BF16 : HQ_DTYPE_FP16, m, k, mode, swizzle, pdl, q.data_ptr(), sf.data_ptr(), dev, st, err, kErrLen);
        }) != 0) {
        Py_RETURN_NONE;
    }
    if (a[4] != Py_None && a[5] != Py_None) return PyTuple_Pack(2, a[4], a[5]);
    return pair_of(q, sf);
    END_HANDLE_TH_ERRORS
}

// rms_norm_quant(input, weight, eps, use_swizzle, use_pdl)
PyObject* rms_norm_quant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    int swizzle, pdl;
    float eps;
    if (nargs != 5 || g_fn.rms == nullptr || at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
    const at::Tensor* const x = plain_tensor(a[0]);
    const at::Tensor* const w = plain_tensor(a[1]);
    if (x == nullptr || w == nullptr || !real(a[2], &eps) || !flag(a[3], &swizzle) || !flag(a[4], &pdl)) Py_RETURN_NONE;
    if (x->scalar_type() != at::kBFloat16 || !quant_input(*x) || x->size(0) == 0) Py_RETURN_NONE;
    const int64_t m = x->size(0), k = x->size(1);
    if (k % 128 != 0 || k <= 0 || k > 8192 || w->dim() != 1 || w->size(0) != k || w->scalar_type() != at::kBFloat16 ||
        !w->is_contiguous() || w->device() != x->device()) {
        Py_RETURN_NONE;
    }
    const int64_t m_sf = swizzle != 0 ? (m + 127) / 128 * 128 : m;
    const void* const px = x->data_ptr();
    const int64_t ld = x->stride(0);
    const void* const pw = w->data_ptr();
    const int dev = x->get_device();
    void* const st = stream_of(*x);
    const auto on_device = at::TensorOptions().device(x->device());
    at::Tensor q, sf;
    if (unlocked([&](char* err) {
            q = at::empty({m, k}, on_device.dtype(at::kFloat8_e4m3fn));
            sf = at::empty({m_sf, k / 32}, on_device.dtype(at::kByte));
            return g_fn.rms(px, ld, pw, eps, m, k, swizzle, pdl, q.data_ptr(), sf.data_ptr(), dev, st, err, kErrLen);
        }) != 0) {
        Py_RETURN_NONE;
    }
    return pair_of(q, sf);
    END_HANDLE_TH_ERRORS
}

// dense_gemm(input, weight, sfa, sfb, output, bias, alpha, sm_count, mode, use_pdl, epilogue, output_sf,
//            situ_beta, situ_linear_beta) -> True, or None when the call is not an ordinary one
PyObject* dense_gemm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    constexpr int kIdentity = HQ_EPILOGUE_IDENTITY, kSigmoid = HQ_EPILOGUE_SIGMOID, kSitu = HQ_EPILOGUE_SITU_QUANT;
    int sm_count, pdl, epilogue;
    if (nargs != 14 || g_fn.dense == nullptr || at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
    const at::Tensor* const x = plain_tensor(a[0]);
    const at::Tensor* const w = plain_tensor(a[1]);
    const at::Tensor* const sfa = plain_tensor(a[2]);
    const at::Tensor* const sfb = plain_tensor(a[3]);
    const at::Tensor* const out = plain_tensor(a[4]);
    const int mode = mode_id(a[8]);
    if (x == nullptr || w == nullptr || sfa == nullptr || sfb == nullptr || out == nullptr || mode < 0 ||
        mode == HQ_MODE_W4A8_MXFP4 || !small_int(a[7], &sm_count) || !small_int(a[9], &pdl) || pdl < 0 || pdl > 2 || !small_int(a[10], &epilogue)) {
        Py_RETURN_NONE;
    }
    const bool fp8 = mode == HQ_MODE_W8A8_MXFP8, nvfp4 = mode == HQ_MODE_W4A4_NVFP4, situ = epilogue == kSitu;
    if (epilogue != kIdentity && epilogue != kSigmoid && !(situ && fp8)) Py_RETURN_NONE;
    if (x->dim() != 2 || w->dim() != 2 || out->dim() != 2 || sfa->dim() < 1 || sfb->dim() < 1) Py_RETURN_NONE;
    if (!bytes(*x) || !bytes(*w) || !u8(*sfa) || !u8(*sfb)) Py_RETURN_NONE;
    const auto dev = x->device();
    if (w->device() != dev || sfa->device() != dev || sfb->device() != dev || out->device() != dev) Py_RETURN_NONE;
    if (!x->is_contiguous() || !w->is_contiguous() || !sfa->is_contiguous() || !sfb->is_contiguous()) Py_RETURN_NONE;
    const int64_t m = x->size(0), n = w->size(0), k = fp8 ? w->size(1) : w->size(1) * 2;
    if (m == 0 || n == 0 || x->size(1) != w->size(1)) Py_RETURN_NONE;
    if (out->size(0) != m || out->size(1) != (situ ? n / 2 : n)) Py_RETURN_NONE;
    const int64_t sf_k = k / (nvfp4 ? 16 : 32), m_sf = (m + 127) / 128 * 128;
    if (sfa->numel() < m_sf * sf_k) Py_RETURN_NONE;
    if (!fp8 && (sfa->size(-1) != sf_k || sfb->size(-1) != sf_k)) Py_RETURN_NONE;
    const void* bias = nullptr;
    if (a[5] != Py_None) {
        const at::Tensor* const b = plain_tensor(a[5]);
        if (!fp8 || (!situ && m % 256 != 0) || b == nullptr || b->scalar_type() != at::kBFloat16 || b->dim() != 1 ||
            b->numel() != n || !b->is_contiguous() || b->device() != dev) {
            Py_RETURN_NONE;
        }
        bias = b->data_ptr();
    }
    const float* alpha = nullptr;
    if (a[6] != Py_None) {
        const at::Tensor* const t = plain_tensor(a[6]);
        if (!nvfp4 || t == nullptr || t->scalar_type() != at::kFloat || t->numel() < 1 || t->device() != dev) Py_RETURN_NONE;
        alpha = static_cast<const float*>(t->data_ptr());
    } else if (nvfp4) {
        Py_RETURN_NONE;
    }
    const void* const px = x->data_ptr();
    const void* const pw = w->data_ptr();
    const void* const psa = sfa->data_ptr();
    const void* const psb = sfb->data_ptr();
    void* const po = out->data_ptr();
    const int64_t na = sfa->numel(), nb = sfb->numel(), ldo = out->stride(0);
    const int d = x->get_device();
    void* const st = stream_of(*x);
    int rc;
    if (situ) {
        float beta, lin = 0.0f;
        const at::Tensor* const osf = plain_tensor(a[11]);
        if (osf == nullptr || !u8(*osf) || !osf->is_contiguous() || osf->device() != dev || !out->is_contiguous() ||
            out->scalar_type() != at::kFloat8_e4m3fn || !real(a[12], &beta) || (a[13] != Py_None && !real(a[13], &lin))) {
            Py_RETURN_NONE;
        }
        void* const pos = osf->data_ptr();
        const int64_t no = osf->numel();
        rc = unlocked_gemm([&](char* err) {
            return g_fn.situ(px, pw, psa, psb, po, pos, bias, m, n, k, na, nb, no, beta, lin, sm_count, pdl != 0 ? 1 : 0, d, st,
                             err, kErrLen);
        });
    } else {
        if (out->scalar_type() != at::kBFloat16 || out->stride(1) != 1) Py_RETURN_NONE;
        rc = unlocked_gemm([&](char* err) {
            return g_fn.dense(px, pw, psa, psb, po, bias, alpha, m, n, k, na, nb, ldo, mode, epilogue, sm_count, pdl, d, st, err,
                              kErrLen);
        });
    }
    if (rc != 0) Py_RETURN_NONE;
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// grouped_gemm(kind, input, weight, sfa, sfb, table, output, bias, alpha, max_m_per_expert, sm_count, mode): kind 2 masked,
// 3 contiguous (whose max_m_per_expert is ignored)
PyObject* grouped_gemm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    int kind, max_m, sm_count;
    if (nargs != 12 || g_fn.masked == nullptr || at::impl::torch_function_mode_enabled()) Py_RETURN_NONE;
    const at::Tensor* const x = plain_tensor(a[1]);
    const at::Tensor* const w = plain_tensor(a[2]);
    const at::Tensor* const sfa = plain_tensor(a[3]);
    const at::Tensor* const sfb = plain_tensor(a[4]);
    const at::Tensor* const table = plain_tensor(a[5]);
    const at::Tensor* const out = plain_tensor(a[6]);
    const int mode = mode_id(a[11]);
    if (x == nullptr || w == nullptr || sfa == nullptr || sfb == nullptr || table == nullptr || out == nullptr || mode < 0 ||
        !small_int(a[0], &kind) || !small_int(a[9], &max_m) || !small_int(a[10], &sm_count)) {
        Py_RETURN_NONE;
    }
    const bool masked = kind == 2, fp8 = mode == HQ_MODE_W8A8_MXFP8, nvfp4 = mode == HQ_MODE_W4A4_NVFP4,
               w4a8 = mode == HQ_MODE_W4A8_MXFP4;
    if (x->dim() != 2 || w->dim() != 3 || table->dim() != 1 || out->dim() != 2 || sfa->dim() < 1 || sfb->dim() < 1) {
        Py_RETURN_NONE;
    }
    if (!bytes(*x) || !bytes(*w) || !u8(*sfa) || !u8(*sfb) || table->scalar_type() != at::kInt) Py_RETURN_NONE;
    const auto dev = x->device();
    if (w->device() != dev || sfa->device() != dev || sfb->device() != dev || out->device() != dev || table->device() != dev) {
        Py_RETURN_NONE;
    }
    const int64_t m = x->size(0), e = w->size(0), n = w->size(1), k = fp8 ? w->size(2) : w->size(2) * 2;
    if (m == 0 || n == 0 || e == 0 || x->size(1) != (w4a8 ? k : w->size(2))) Py_RETURN_NONE;
    if (masked ? (max_m <= 0 || m != e * int64_t(max_m) || table->size(0) != e) : table->size(0) != m) Py_RETURN_NONE;
    if (out->size(0) != m || out->size(1) != n || out->scalar_type() != at::kBFloat16 || out->stride(1) != 1) Py_RETURN_NONE;
    if (!x->is_contiguous() || !w->is_contiguous() || !sfa->is_contiguous() || !sfb->is_contiguous() ||
        !table->is_contiguous()) {
        Py_RETURN_NONE;
    }
    const int64_t sf_k = k / (nvfp4 ? 16 : 32);
    if (!fp8 && (sfa->size(-1) != sf_k || sfb->size(-1) != sf_k)) Py_RETURN_NONE;
    const void* bias = nullptr;
    if (a[7] != Py_None) {
        const at::Tensor* const b = plain_tensor(a[7]);
        if (!fp8 || b == nullptr || b->scalar_type() != at::kBFloat16 || b->numel() != e * n || !b->is_contiguous() ||
            b->device() != dev) {
            Py_RETURN_NONE;
        }
        bias = b->data_ptr();
    }
    const float* alpha = nullptr;
    if (a[8] != Py_None) {
        const at::Tensor* const t = plain_tensor(a[8]);
        if (!nvfp4 || t == nullptr || t->scalar_type() != at::kFloat || t->numel() != e || !t->is_contiguous() ||
            t->device() != dev) {
            Py_RETURN_NONE;
        }
        alpha = static_cast<const float*>(t->data_ptr());
    } else if (nvfp4) {
        Py_RETURN_NONE;
    }
    const void* const px = x->data_ptr();
    const void* const pw = w->data_ptr();
    const void* const psa = sfa->data_ptr();
    const void* const psb = sfb->data_ptr();
    const int32_t* const pt = static_cast<const int32_t*>(table->data_ptr());
    void* const po = out->data_ptr();
    const int64_t na = sfa->numel(), nb = sfb->numel(), ldo = out->stride(0);
    const int d = x->get_device();
    void* const st = stream_of(*x);
    const int rc = unlocked_gemm([&](char* err) {
        // the shape rules that the wrapper asks for first
        if (g_fn.describe_group(kind, e, masked ? max_m : m / e, m, n, k, mode, 148, -1, err, kErrLen) != 0) return 1;
        return (masked ? g_fn.masked : g_fn.contiguous)(px, pw, psa, psb, pt, po, bias, alpha, e, masked ? max_m : m, n, k, na,
                                                        nb, ldo, mode, sm_count, 1, d, st, err, kErrLen);
    });
    if (rc != 0) Py_RETURN_NONE;
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// bind(quant, rms, dense, situ, describe_group, masked, contiguous, hold_switches): addresses of the C ABI's entry points
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long p[8];
    if (!PyArg_ParseTuple(args, "KKKKKKKK", &p[0], &p[1], &p[2], &p[3], &p[4], &p[5], &p[6], &p[7])) return nullptr;
    g_fn.quant = reinterpret_cast<QuantFn>(p[0]);
    g_fn.rms = reinterpret_cast<RmsFn>(p[1]);
    g_fn.dense = reinterpret_cast<DenseFn>(p[2]);
    g_fn.situ = reinterpret_cast<SituFn>(p[3]);
    g_fn.describe_group = reinterpret_cast<DescribeGroupFn>(p[4]);
    g_fn.masked = reinterpret_cast<MaskedFn>(p[5]);
    g_fn.contiguous = reinterpret_cast<ContiguousFn>(p[6]);
    g_fn.hold_switches = reinterpret_cast<decltype(&hq_hold_switches)>(p[7]);
    Py_RETURN_NONE;
}

template <typename F>
PyCFunction method(F f) {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef methods[] = {{"group_wise_quant", method(group_wise_quant), METH_FASTCALL, nullptr},
                         {"rms_norm_quant", method(rms_norm_quant), METH_FASTCALL, nullptr},
                         {"dense_gemm", method(dense_gemm), METH_FASTCALL, nullptr},
                         {"grouped_gemm", method(grouped_gemm), METH_FASTCALL, nullptr},
                         {"bind", bind, METH_VARARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "halops_b200_fast_path", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_halops_b200_fast_path() { return PyModule_Create(&module); }
