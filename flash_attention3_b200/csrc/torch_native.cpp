// Native half of the torch front end (ops.py, torch_binding.py): checks, allocations, the parameter
// block and the call into the C ABI, in one C++ function per entry point.
//
// What bounds a small call is host time.  Filling the parameter block and its pointers through
// ctypes, three or four torch.empty calls, a device context manager and the tensor checks in Python
// took 41-50 us per ops.fa3_bwd (27-35 us per ops.fa3_fwd) against 18 us of GPU time for one head of
// 1024 rows; a forward + gradient through autograd took 225-249 us of host time, most of it in two
// torch.library.custom_op wrappers.  The same steps here cost a few microseconds on top of the
// kernel launches.
//
// Two front doors share the functions below: CPython fast calls for ops.py, and the dispatcher ops
// fa3b200::attention_fwd / attention_bwd with a C++ autograd function over them for torch_binding.py.
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/library.h>
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstring>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "shaobo_fa3_api.h"
#include "shaobo_fa3_b200_ext.h"
#include "shaobo_fa3_components.h"

namespace {

using at::Tensor;

// A status other than SUCCESS from the C ABI: ops.py turns it into Fa3Error.
struct AbiError {
    const char* entry;
    int code;
};

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
    return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}
Tensor like(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t.device()); }

void require_cuda(std::initializer_list<const Tensor*> tensors) {
    for (const Tensor* t : tensors) {
        if (!t->defined()) continue;
        TORCH_CHECK(t->is_cuda(), "flash_attention3_b200 has no CPU path: tensors must live on a CUDA device");
        TORCH_CHECK(t->is_contiguous(), "contiguous tensors are required ([B,H,S,D] or [B,S,H,D])");
    }
}

int32_t dtype_code(const Tensor& q) {
    if (q.scalar_type() == at::kHalf) return SHAOBO_FA3_DTYPE_FP16;
    TORCH_CHECK_TYPE(q.scalar_type() == at::kBFloat16, "unsupported dtype ", q.scalar_type(), ": fp16 or bf16");
    return SHAOBO_FA3_DTYPE_BF16;
}

bool is_bshd(const char* layout) {
    if (std::strcmp(layout, "bshd") == 0) return true;
    TORCH_CHECK_VALUE(std::strcmp(layout, "bhsd") == 0, "unknown layout '", layout, "'");
    return false;
}

void same_kind(const char* name, const Tensor& t, const Tensor& q) {
    TORCH_CHECK_TYPE(t.scalar_type() == q.scalar_type() && t.device() == q.device(), name, " must have the dtype and device of q");
}

// Shapes, dtypes and devices of one fixed-length problem (the C ABI takes raw pointers, so a tensor of
// the wrong size would be read or written out of bounds), and the parameter block that describes it.
struct Options {
    int64_t causal = 0;  // (flags other than 0 and 1 are turned away by the C ABI)
    std::optional<double> scale;
    bool bshd = false;
    int64_t window_left = -1, window_right = -1;
    Tensor seqused_q, seqused_k;
    double softcap = 0.0;
    int64_t deterministic = 0;
    int64_t sync = 0;
};

void set_common(ShaoboFa3Params* p, const Tensor& q, const Options& o) {
    p->causal = int32_t(o.causal);
    p->dtype = dtype_code(q);
    p->deterministic = int32_t(o.deterministic);
    p->sync_after_launch = int32_t(o.sync);
    p->window_left = int32_t(o.window_left);
    p->window_right = int32_t(o.window_right);
    p->softcap = float(o.softcap);
    if (o.scale.has_value()) {
        p->softmax_scale = float(*o.scale);
        p->softmax_scale_is_set = 1;
    }
}

const int32_t* seqused_ptr(const Tensor& t) {
    if (!t.defined()) return nullptr;
    TORCH_CHECK_TYPE(t.scalar_type() == at::kInt && t.is_cuda(), "seqused must be an int32 CUDA tensor");
    return t.const_data_ptr<int32_t>();
}

ShaoboFa3Params fixed_problem(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& dout,
                              const Tensor& lse, const Options& o) {
    TORCH_CHECK_VALUE(q.dim() == 4 && k.dim() == 4, "q and k must be 4-D ([B,H,S,D] or [B,S,H,D])");
    ShaoboFa3Params p;
    shaobo_fa3_params_init(&p);
    set_common(&p, q, o);
    TORCH_CHECK_VALUE(v.sizes() == k.sizes(), "v ", v.sizes(), " must have the shape of k ", k.sizes());
    const int head_dim = o.bshd ? 2 : 1, row_dim = o.bshd ? 1 : 2;
    const int64_t hq = q.size(head_dim), hkv = k.size(head_dim), sq = q.size(row_dim);
    TORCH_CHECK_VALUE(q.size(0) == k.size(0) && q.size(3) == k.size(3) && hkv != 0 && hq % hkv == 0, "q ", q.sizes(),
                      " and k ", k.sizes(), " do not describe one problem");
    same_kind("k", k, q);
    same_kind("v", v, q);
    for (const auto& [name, t] : {std::pair<const char*, const Tensor*>{"out", &out}, {"dout", &dout}}) {
        if (!t->defined()) continue;
        same_kind(name, *t, q);
        TORCH_CHECK_VALUE(t->sizes() == q.sizes(), name, " ", t->sizes(), " must have the shape of q ", q.sizes());
    }
    if (lse.defined()) {
        TORCH_CHECK_TYPE(lse.scalar_type() == at::kFloat && lse.device() == q.device(), "softmax_lse must be fp32 on the device of q");
        TORCH_CHECK_VALUE(lse.dim() == 3 && lse.size(0) == q.size(0) && lse.size(1) == hq && lse.size(2) == sq, "softmax_lse ",
                          lse.sizes(), " must be [B,Hq,Sq] = (", q.size(0), ", ", hq, ", ", sq, ")");
    }
    p.batch = int32_t(q.size(0));
    p.seqlen_q = int32_t(sq);
    p.seqlen_k = int32_t(k.size(row_dim));
    p.num_heads_q = int32_t(hq);
    p.num_heads_kv = int32_t(hkv);
    p.head_dim_qk = p.head_dim_v = int32_t(q.size(3));
    p.layout = o.bshd ? SHAOBO_FA3_LAYOUT_BSHD : SHAOBO_FA3_LAYOUT_BHSD;
    p.seqused_q = seqused_ptr(o.seqused_q);
    p.seqused_k = seqused_ptr(o.seqused_k);
    return p;
}

ShaoboFa3Params packed_problem(const Tensor& q, const Tensor& k, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q,
                               int64_t max_k, const Options& o) {
    TORCH_CHECK_TYPE(cu_q.scalar_type() == at::kInt && cu_k.scalar_type() == at::kInt, "cu_seqlens must be int32");
    TORCH_CHECK_VALUE(q.dim() == 3 && k.dim() == 3, "q and k must be 3-D ([total,H,D])");
    ShaoboFa3Params p;
    shaobo_fa3_params_init(&p);
    set_common(&p, q, o);
    p.batch = int32_t(cu_q.numel() - 1);
    p.seqlen_q = p.max_seqlen_q = int32_t(max_q);
    p.seqlen_k = p.max_seqlen_k = int32_t(max_k);
    p.num_heads_q = int32_t(q.size(1));
    p.num_heads_kv = int32_t(k.size(1));
    p.head_dim_qk = p.head_dim_v = int32_t(q.size(2));
    p.layout = SHAOBO_FA3_LAYOUT_BSHD;
    p.cu_seqlens_q = cu_q.const_data_ptr<int32_t>();
    p.cu_seqlens_k = cu_k.const_data_ptr<int32_t>();
    p.total_q = q.size(0);
    p.total_k = k.size(0);
    return p;
}

std::tuple<Tensor, Tensor> run_forward(ShaoboFa3Params& p, const Tensor& q, const Tensor& k, const Tensor& v, Tensor lse) {
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    Tensor out = like(q);
    p.reserved_ptr[SHAOBO_FA3_RESERVED_PTR_STREAM] = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const int code = shaobo_fa3_b200_fwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), out.data_ptr(), lse.data_ptr(), &p);
    if (code != SHAOBO_FA3_STATUS_SUCCESS) throw AbiError{"shaobo_fa3_b200_fwd", code};
    return {std::move(out), std::move(lse)};
}

struct Gradients {
    Tensor dq, dk, dv;
};
Gradients run_backward(ShaoboFa3Params& p, const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v,
                       const Tensor& out, const Tensor& lse, Tensor workspace, Gradients g, const Tensor& delta) {
    const size_t need = shaobo_fa3_bwd_v2_workspace_bytes(&p);
    if (need == 0) throw AbiError{"shaobo_fa3_bwd_v2_validate", shaobo_fa3_bwd_v2_validate(&p)};
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    if (!workspace.defined() || workspace.nbytes() < need) workspace = empty({int64_t(need)}, at::kByte, q.device());
    p.workspace = workspace.data_ptr();
    p.workspace_bytes = workspace.nbytes();
    if (!g.dq.defined()) g = Gradients{like(q), like(k), like(v)};
    p.reserved_ptr[SHAOBO_FA3_RESERVED_PTR_STREAM] = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const int code = shaobo_fa3_bwd_v2(dout.const_data_ptr(), q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(),
                                       out.const_data_ptr(), lse.const_data_ptr(), g.dq.data_ptr(), g.dk.data_ptr(),
                                       g.dv.data_ptr(), delta.defined() ? delta.data_ptr() : nullptr, &p);
    if (code != SHAOBO_FA3_STATUS_SUCCESS) throw AbiError{"shaobo_fa3_bwd_v2", code};
    return g;
}

// ------------------------------------------------------------------ CPython front door (ops.py)
Tensor arg_tensor(PyObject* o, const char* name) {
    if (o == Py_None) return Tensor();
    TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor");
    return THPVariable_Unpack(o);
}
Tensor arg_required(PyObject* o, const char* name) {
    Tensor t = arg_tensor(o, name);
    TORCH_CHECK_TYPE(t.defined(), name, " must be a tensor");
    return t;
}
bool arg_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
// bool of a torch schema: None, or what says by itself whether it is true (a string does not)
bool arg_schema_bool(PyObject* o, const char* name) {
    const PyNumberMethods* number = Py_TYPE(o)->tp_as_number;
    TORCH_CHECK_TYPE(o == Py_None || (number != nullptr && number->nb_bool != nullptr), name, " must be a bool");
    return arg_bool(o);
}
// (the conversions of ints, bools, floats and tuples, what nearly every call passes, need no object of their own)
int64_t long_value(PyObject* i) {
    const long long v = PyLong_AsLongLong(i);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
int64_t arg_int(PyObject* o) {  // int(o)
    if (PyLong_CheckExact(o) || PyBool_Check(o)) return long_value(o);
    THPObjectPtr i(PyNumber_Long(o));
    if (!i) throw python_error();
    return long_value(i.get());
}
int64_t arg_schema_int(PyObject* o) {  // (no float)
    if (PyLong_CheckExact(o)) return long_value(o);
    THPObjectPtr i(PyNumber_Index(o));
    if (!i) throw python_error();
    return long_value(i.get());
}
double arg_double(PyObject* o) {  // a number
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
}
double arg_float(PyObject* o) {  // float(o)
    if (PyFloat_CheckExact(o)) return PyFloat_AS_DOUBLE(o);
    const THPObjectPtr f(PyNumber_Float(o));
    if (!f) throw python_error();
    return PyFloat_AS_DOUBLE(f.get());
}
const char* arg_str(PyObject* o) {
    const char* s = PyUnicode_AsUTF8(o);
    if (s == nullptr) throw python_error();
    return s;
}
void arg_window(PyObject* o, Options* opt) {  // int(o[0]), int(o[1])
    if (PyTuple_CheckExact(o) && PyTuple_GET_SIZE(o) >= 2) {
        opt->window_left = arg_int(PyTuple_GET_ITEM(o, 0));
        opt->window_right = arg_int(PyTuple_GET_ITEM(o, 1));
        return;
    }
    for (const long i : {0, 1}) {
        const THPObjectPtr index(PyLong_FromLong(i));
        THPObjectPtr item(index ? PyObject_GetItem(o, const_cast<PyObject*>(index.get())) : nullptr);
        if (!item) throw python_error();
        (i == 0 ? opt->window_left : opt->window_right) = arg_int(item.get());
    }
}
void arg_count(Py_ssize_t got, Py_ssize_t want) { TORCH_CHECK_TYPE(got == want, "expected ", want, " arguments, got ", got); }

// (entry, code) of a call that the C ABI refused
PyObject* refused(const AbiError& e) { return Py_BuildValue("(si)", e.entry, e.code); }

PyObject* pack(std::initializer_list<const Tensor*> tensors) {
    PyObject* out = PyTuple_New(Py_ssize_t(tensors.size()));
    if (out == nullptr) throw python_error();
    Py_ssize_t i = 0;
    for (const Tensor* t : tensors) PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(*t));
    return out;
}

// fwd(q, k, v, causal, scale, layout, window, sync, seqused_q, seqused_k, softcap)
PyObject* py_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 11);
    const Tensor q = arg_required(a[0], "q"), k = arg_required(a[1], "k"), v = arg_required(a[2], "v");
    require_cuda({&q, &k, &v});
    Options o;
    o.causal = arg_int(a[3]);
    if (a[4] != Py_None) o.scale = arg_float(a[4]);
    o.bshd = is_bshd(arg_str(a[5]));
    arg_window(a[6], &o);
    o.sync = arg_int(a[7]);
    o.seqused_q = arg_tensor(a[8], "seqused_q");
    o.seqused_k = arg_tensor(a[9], "seqused_k");
    o.softcap = arg_float(a[10]);
    ShaoboFa3Params p = fixed_problem(q, k, v, Tensor(), Tensor(), Tensor(), o);
    try {
        Tensor out, lse;
        {
            pybind11::gil_scoped_release no_gil;  // (as around a ctypes call; with sync the call waits)
            std::tie(out, lse) = run_forward(p, q, k, v, empty({p.batch, p.num_heads_q, p.seqlen_q}, at::kFloat, q.device()));
        }
        return pack({&out, &lse});
    } catch (const AbiError& e) {
        return refused(e);
    }
    END_HANDLE_TH_ERRORS
}

// bwd(dout, q, k, v, out, lse, causal, scale, deterministic, workspace, return_delta, sync, layout, window,
//     seqused_q, seqused_k, outputs, softcap)
PyObject* py_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 18);
    const Tensor dout = arg_required(a[0], "dout"), q = arg_required(a[1], "q"), k = arg_required(a[2], "k"),
                 v = arg_required(a[3], "v"), out = arg_required(a[4], "out"), lse = arg_required(a[5], "softmax_lse");
    require_cuda({&dout, &q, &k, &v, &out, &lse});
    Options o;
    o.causal = arg_int(a[6]);
    if (a[7] != Py_None) o.scale = arg_float(a[7]);
    o.deterministic = arg_int(a[8]);
    const Tensor workspace = arg_tensor(a[9], "workspace");
    const bool return_delta = arg_bool(a[10]);
    o.sync = arg_int(a[11]);
    o.bshd = is_bshd(arg_str(a[12]));
    arg_window(a[13], &o);
    o.seqused_q = arg_tensor(a[14], "seqused_q");
    o.seqused_k = arg_tensor(a[15], "seqused_k");
    o.softcap = arg_float(a[17]);
    ShaoboFa3Params p = fixed_problem(q, k, v, out, dout, lse, o);
    Gradients g;
    if (a[16] != Py_None) {
        PyObject* seq = PySequence_Fast(a[16], "outputs must be (dq, dk, dv)");
        if (seq == nullptr) throw python_error();
        const bool three = PySequence_Fast_GET_SIZE(seq) == 3;
        if (three) {
            g = Gradients{arg_required(PySequence_Fast_GET_ITEM(seq, 0), "dq"), arg_required(PySequence_Fast_GET_ITEM(seq, 1), "dk"),
                          arg_required(PySequence_Fast_GET_ITEM(seq, 2), "dv")};
        }
        Py_DECREF(seq);
        TORCH_CHECK_VALUE(three, "outputs must be (dq, dk, dv)");
        require_cuda({&g.dq, &g.dk, &g.dv});
        for (const auto& [t, like] : {std::pair<const Tensor*, const Tensor*>{&g.dq, &q}, {&g.dk, &k}, {&g.dv, &v}}) {
            TORCH_CHECK_VALUE(t->sizes() == like->sizes() && t->scalar_type() == like->scalar_type() && t->device() == like->device(),
                              "outputs must match q, k, v in shape, dtype and device");
        }
    }
    try {
        Tensor delta;
        {
            pybind11::gil_scoped_release no_gil;
            if (return_delta) delta = empty({p.batch, p.num_heads_q, p.seqlen_q}, at::kFloat, q.device());
            g = run_backward(p, dout, q, k, v, out, lse, workspace, std::move(g), delta);
        }
        return return_delta ? pack({&g.dq, &g.dk, &g.dv, &delta}) : pack({&g.dq, &g.dk, &g.dv});
    } catch (const AbiError& e) {
        return refused(e);
    }
    END_HANDLE_TH_ERRORS
}

// fwd_packed(q, k, v, cu_q, cu_k, max_q, max_k, causal, scale, window, sync)
PyObject* py_fwd_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 11);
    const Tensor q = arg_required(a[0], "q"), k = arg_required(a[1], "k"), v = arg_required(a[2], "v"),
                 cu_q = arg_required(a[3], "cu_seqlens_q"), cu_k = arg_required(a[4], "cu_seqlens_k");
    require_cuda({&q, &k, &v, &cu_q, &cu_k});
    Options o;
    o.causal = arg_int(a[7]);
    if (a[8] != Py_None) o.scale = arg_float(a[8]);
    arg_window(a[9], &o);
    o.sync = arg_int(a[10]);
    ShaoboFa3Params p = packed_problem(q, k, cu_q, cu_k, arg_int(a[5]), arg_int(a[6]), o);
    try {
        Tensor out, lse;
        {
            pybind11::gil_scoped_release no_gil;
            std::tie(out, lse) = run_forward(p, q, k, v, empty({q.size(1), q.size(0)}, at::kFloat, q.device()));
        }
        return pack({&out, &lse});
    } catch (const AbiError& e) {
        return refused(e);
    }
    END_HANDLE_TH_ERRORS
}

// bwd_packed(dout, q, k, v, out, lse, cu_q, cu_k, max_q, max_k, causal, scale, deterministic, window, return_delta, sync)
PyObject* py_bwd_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 16);
    const Tensor dout = arg_required(a[0], "dout"), q = arg_required(a[1], "q"), k = arg_required(a[2], "k"),
                 v = arg_required(a[3], "v"), out = arg_required(a[4], "out"), lse = arg_required(a[5], "softmax_lse"),
                 cu_q = arg_required(a[6], "cu_seqlens_q"), cu_k = arg_required(a[7], "cu_seqlens_k");
    require_cuda({&dout, &q, &k, &v, &out, &lse, &cu_q, &cu_k});
    Options o;
    o.causal = arg_int(a[10]);
    if (a[11] != Py_None) o.scale = arg_float(a[11]);
    o.deterministic = arg_int(a[12]);
    arg_window(a[13], &o);
    const bool return_delta = arg_bool(a[14]);
    o.sync = arg_int(a[15]);
    ShaoboFa3Params p = packed_problem(q, k, cu_q, cu_k, arg_int(a[8]), arg_int(a[9]), o);
    try {
        Tensor delta;
        Gradients g;
        {
            pybind11::gil_scoped_release no_gil;
            if (return_delta) delta = empty({q.size(1), q.size(0)}, at::kFloat, q.device());
            g = run_backward(p, dout, q, k, v, out, lse, Tensor(), Gradients{}, delta);
        }
        return return_delta ? pack({&g.dq, &g.dk, &g.dv, &delta}) : pack({&g.dq, &g.dk, &g.dv});
    } catch (const AbiError& e) {
        return refused(e);
    }
    END_HANDLE_TH_ERRORS
}

// ----------------------------------------------------------- dispatcher ops (torch_binding.py)
PyObject* g_error_type = nullptr;  // ops.Fa3Error, for the life of the process

PyObject* py_set_error_type(PyObject*, PyObject* type) {
    Py_INCREF(type);
    Py_XSETREF(g_error_type, type);
    Py_RETURN_NONE;
}

// A call that the C ABI refused raises ops.Fa3Error, through the dispatcher and the autograd engine as well.
[[noreturn]] void fail(const AbiError& e) {
    TORCH_CHECK(g_error_type != nullptr, e.entry, " returned ", e.code, " (", shaobo_fa3_status_string(e.code), ")");
    pybind11::gil_scoped_acquire gil;
    THPObjectPtr error(PyObject_CallFunction(g_error_type, "si", e.entry, e.code));
    if (error) PyErr_SetObject(g_error_type, error.get());
    python_error raised;
    raised.persist();
    throw raised;
}

// (the kernels read dense tensors: strided views are copied)
std::tuple<Tensor, Tensor> attention_fwd(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, bool causal, double scale,
                                         c10::SymInt window_left, c10::SymInt window_right, double softcap, c10::string_view layout) {
    const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous();
    require_cuda({&q, &k, &v});
    Options o;
    o.causal = causal;
    o.scale = scale;
    o.bshd = is_bshd(std::string(layout).c_str());
    o.window_left = window_left.guard_int(__FILE__, __LINE__);
    o.window_right = window_right.guard_int(__FILE__, __LINE__);
    o.softcap = softcap;
    ShaoboFa3Params p = fixed_problem(q, k, v, Tensor(), Tensor(), Tensor(), o);
    try {
        return run_forward(p, q, k, v, empty({p.batch, p.num_heads_q, p.seqlen_q}, at::kFloat, q.device()));
    } catch (const AbiError& e) {
        fail(e);
    }
}

std::tuple<Tensor, Tensor, Tensor> attention_bwd(const Tensor& dout_in, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                                                 const Tensor& out_in, const Tensor& lse_in, bool causal, double scale,
                                                 bool deterministic, c10::SymInt window_left, c10::SymInt window_right,
                                                 double softcap, c10::string_view layout) {
    const Tensor dout = dout_in.contiguous(), q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous(),
                 out = out_in.contiguous(), lse = lse_in.contiguous();
    require_cuda({&dout, &q, &k, &v, &out, &lse});
    Options o;
    o.causal = causal;
    o.scale = scale;
    o.deterministic = deterministic;
    o.bshd = is_bshd(std::string(layout).c_str());
    o.window_left = window_left.guard_int(__FILE__, __LINE__);
    o.window_right = window_right.guard_int(__FILE__, __LINE__);
    o.softcap = softcap;
    ShaoboFa3Params p = fixed_problem(q, k, v, out, dout, lse, o);
    try {
        Gradients g = run_backward(p, dout, q, k, v, out, lse, Tensor(), Gradients{}, Tensor());
        return {std::move(g.dq), std::move(g.dk), std::move(g.dv)};
    } catch (const AbiError& e) {
        fail(e);
    }
}

// Autograd over the two ops.  The ops are reached through the dispatcher, so a call on fake tensors
// runs their fake implementations.
using FwdSignature = std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, bool, double, c10::SymInt, c10::SymInt,
                                                double, c10::string_view);
using BwdSignature = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                        const Tensor&, bool, double, bool, c10::SymInt, c10::SymInt, double,
                                                        c10::string_view);

class Attention : public torch::autograd::Function<Attention> {
  public:
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                          bool causal, double scale, bool deterministic, int64_t window_left, int64_t window_right, double softcap,
                          std::string layout) {
        static const auto op =
            c10::Dispatcher::singleton().findSchemaOrThrow("fa3b200::attention_fwd", "").typed<FwdSignature>();
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        // strided inputs (a transposed view, say) are made dense once, here, and the dense copies are what
        // the backward gets; autograd maps the dense gradients back onto the views
        const Tensor q = q_in.contiguous(), k = k_in.contiguous(), v = v_in.contiguous();
        auto [out, lse] = op.call(q, k, v, causal, scale, window_left, window_right, softcap, layout);
        ctx->save_for_backward({q, k, v, out, lse});
        ctx->saved_data["causal"] = causal;
        ctx->saved_data["scale"] = scale;
        ctx->saved_data["deterministic"] = deterministic;
        ctx->saved_data["window_left"] = window_left;
        ctx->saved_data["window_right"] = window_right;
        ctx->saved_data["softcap"] = softcap;
        ctx->saved_data["layout"] = std::move(layout);
        return out;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        static const auto op =
            c10::Dispatcher::singleton().findSchemaOrThrow("fa3b200::attention_bwd", "").typed<BwdSignature>();
        const auto saved = ctx->get_saved_variables();
        auto& d = ctx->saved_data;
        // with create_graph the op goes through its Autograd kernel, which refuses a second derivative
        std::optional<at::AutoDispatchBelowADInplaceOrView> below_autograd;
        if (!at::GradMode::is_enabled()) below_autograd.emplace();
        auto [dq, dk, dv] = op.call(grads[0], saved[0], saved[1], saved[2], saved[3], saved[4], d["causal"].toBool(),
                                    d["scale"].toDouble(), d["deterministic"].toBool(), d["window_left"].toInt(),
                                    d["window_right"].toInt(), d["softcap"].toDouble(), d["layout"].toStringRef());
        return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// attention(q, k, v, causal, scale, deterministic, window, softcap, layout)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 9);
    const Tensor q = arg_required(a[0], "q"), k = arg_required(a[1], "k"), v = arg_required(a[2], "v");
    // (what the schema of the ops takes)
    const bool causal = arg_schema_bool(a[3], "causal"), deterministic = arg_schema_bool(a[5], "deterministic");
    const double scale = a[4] != Py_None ? arg_double(a[4]) : 1.0 / std::sqrt(double(q.size(-1)));
    THPObjectPtr window(PySequence_Tuple(a[6]));
    if (!window) throw python_error();
    int64_t sides[2];
    for (const int i : {0, 1}) {
        PyObject* item = PyTuple_GetItem(window.get(), i);
        if (item == nullptr) throw python_error();
        sides[i] = arg_schema_int(item);
    }
    const double softcap = arg_float(a[7]);
    const std::string layout = arg_str(a[8]);
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = Attention::apply(q, k, v, causal, scale, deterministic, sides[0], sides[1], softcap, layout);
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

template <PyObject* (*fn)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn));
}

PyMethodDef kMethods[] = {
    {"fwd", fast<py_fwd>(), METH_FASTCALL, nullptr},
    {"bwd", fast<py_bwd>(), METH_FASTCALL, nullptr},
    {"fwd_packed", fast<py_fwd_packed>(), METH_FASTCALL, nullptr},
    {"bwd_packed", fast<py_bwd_packed>(), METH_FASTCALL, nullptr},
    {"attention", fast<py_attention>(), METH_FASTCALL, nullptr},
    {"set_error_type", py_set_error_type, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

TORCH_LIBRARY(fa3b200, m) {
    // (with a fake implementation and dense results the ops are fit for torch.compile, also where it takes no others)
    const std::vector<at::Tag> tags = {at::Tag::pt2_compliant_tag};
    m.def(
        "attention_bwd(Tensor dout, Tensor q, Tensor k, Tensor v, Tensor out, Tensor softmax_lse, bool causal, "
        "float softmax_scale, bool deterministic, SymInt window_left=-1, SymInt window_right=-1, float softcap=0.0, "
        "str layout=\"bhsd\") -> (Tensor, Tensor, Tensor)",
        tags);
    m.def(
        "attention_fwd(Tensor q, Tensor k, Tensor v, bool causal, float softmax_scale, SymInt window_left=-1, "
        "SymInt window_right=-1, float softcap=0.0, str layout=\"bhsd\") -> (Tensor, Tensor)",
        tags);
}
TORCH_LIBRARY_IMPL(fa3b200, CUDA, m) {
    m.impl("attention_bwd", attention_bwd);
    m.impl("attention_fwd", attention_fwd);
}
// The ops themselves have no derivative (attention() has one, of first order): differentiating them raises.
// Without these kernels torch warns and leaves their part of the gradient out.
TORCH_LIBRARY_IMPL(fa3b200, Autograd, m) {
    m.impl("attention_bwd", torch::autograd::autogradNotImplementedFallback());
    m.impl("attention_fwd", torch::autograd::autogradNotImplementedFallback());
}

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&kModule); }
