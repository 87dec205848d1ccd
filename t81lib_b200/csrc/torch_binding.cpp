// Host path of the Python layer in native code: the calls that run once per Linear or per training step check their
// tensors, allocate results and scratch through torch's caching allocator and enter the C ABI from here.  A decode-sized
// product runs a few microseconds on the device; the same steps in Python (ctypes with sixteen arguments, attribute
// reads, torch.empty) took 14 of them per call.
//
// Nothing is computed here.  Calls that need a conversion, a copy or an autograd node return None and are taken by the
// general path in Python.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <optional>

#include "../../include/t81_b200.h"

namespace {

using at::Tensor;

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return T81B200_F32;
        case at::kBFloat16: return T81B200_BF16;
        case at::kHalf: return T81B200_F16;
        default: return -1;
    }
}

// A return code of the library as the exception the Python layer raises for it (t81lib_b200._capi.check).
struct LibraryError {
    int code;
};
void check(int code) {
    if (code != T81B200_OK) throw LibraryError{code};
}
PyObject *raise_library_error(int code) {
    PyObject *mod = PyImport_ImportModule("t81lib_b200._capi");
    if (mod) {
        PyObject *r = PyObject_CallMethod(mod, "check", "i", code);
        Py_XDECREF(r);
        Py_DECREF(mod);
    }
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "t81_b200 error %d", code);
    return nullptr;
}

// The library's failures inside autograd travel as the Python exception they stand for: a backward runs in a worker thread of
// torch's, which carries std::exceptions to the caller and ends the process on anything else.
template <typename F> auto as_python_error(F &&f) {
    try {
        return f();
    } catch (const LibraryError &e) {
        const PyGILState_STATE gil = PyGILState_Ensure();
        raise_library_error(e.code);
        python_error error;
        error.persist();
        PyGILState_Release(gil);
        throw error;
    }
}

const float *float_ptr(const std::optional<Tensor> &t) { return t ? t->const_data_ptr<float>() : nullptr; }

bool float_vector(const Tensor &t, const c10::Device &device, int64_t n) {
    return t.scalar_type() == at::kFloat && t.device() == device && t.is_contiguous() && t.numel() == n;
}

void *stream_of(const c10::Device &device) { return c10::cuda::getCurrentCUDAStream(device.index()).stream(); }

// Makes the tensors' device current where it is not.
struct OnDevice {
    std::optional<c10::cuda::CUDAGuard> guard;
    explicit OnDevice(const c10::Device &device) {
        if (c10::cuda::current_device() != device.index()) guard.emplace(device);
    }
};

// x as token-major rows: (tokens, k) or (batch, tokens, k) with unit column stride and one distance between rows.
struct Rows {
    const void *data = nullptr;
    int64_t tokens = 0, ld = 0;
    int dtype = -1;
};
bool as_rows(const Tensor &x, int64_t k, Rows &r) {
    const auto dim = x.dim();
    if ((dim != 2 && dim != 3) || x.size(dim - 1) != k || (k > 1 && x.stride(dim - 1) != 1)) return false;
    r.dtype = dtype_code(x.scalar_type());
    if (r.dtype < 0) return false;
    r.tokens = dim == 2 ? x.size(0) : x.size(0) * x.size(1);
    r.ld = x.stride(dim - 2);
    if (dim == 3 && x.size(0) > 1) {
        if (x.size(1) == 1) r.ld = x.stride(0);
        else if (x.stride(0) != x.size(1) * x.stride(1)) return false;
    }
    if (r.tokens <= 1) r.ld = k;
    r.data = x.const_data_ptr();
    return r.ld >= k;
}

Tensor product(const Tensor &t2, int64_t rows, int64_t k, const float *row_scale, const float *bias, const Rows &x, c10::IntArrayRef shape,
               at::ScalarType out_type, const c10::Device &device, int fp32_planes) {
    OnDevice on(device);
    Tensor y = at::empty(shape, at::TensorOptions().dtype(out_type).device(device));
    if (x.tokens == 0) return y;
    const size_t need = t81b200_linear_t2_workspace_bytes(x.data, x.dtype, x.ld, rows, x.tokens, k, fp32_planes);
    Tensor ws;
    if (need) ws = at::empty({(int64_t)need}, at::TensorOptions().dtype(at::kByte).device(device));
    check(t81b200_linear_t2(t2.const_data_ptr<uint8_t>(), row_scale, bias, y.mutable_data_ptr(), rows, x.data, x.dtype, x.ld, dtype_code(out_type), rows,
                            x.tokens, k, 1.0f, 0.0f, fp32_planes, need ? ws.mutable_data_ptr() : nullptr, need, stream_of(device)));
    return y;
}

// ---- Product(t2, rows, k, row_scale): a weight in the decode-stream layout, called with (x, bias=None, out_dtype=None) ----

struct ProductObject {
    PyObject_HEAD
    vectorcallfunc call;
    Tensor *t2, *row_scale;  // row_scale: null where the weight has none
    int64_t rows, k;
};

bool plain_tensor(PyObject *o) { return THPVariable_CheckExact(o); }

PyObject *product_call(PyObject *self, PyObject *const *args, size_t nargsf, PyObject *kwnames) {
    HANDLE_TH_ERRORS
    auto *p = reinterpret_cast<ProductObject *>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if (kwnames && PyTuple_GET_SIZE(kwnames)) {
        PyErr_SetString(PyExc_TypeError, "Product takes positional arguments (x, bias, out_dtype)");
        return nullptr;
    }
    if (n < 1 || !plain_tensor(args[0])) Py_RETURN_NONE;
    const Tensor &x = THPVariable_Unpack(args[0]);
    const c10::Device device = p->t2->device();
    Rows rows;
    if (x.device() != device || x.layout() != at::kStrided || !as_rows(x, p->k, rows)) Py_RETURN_NONE;
    const bool grad = at::GradMode::is_enabled();
    if (grad && x.requires_grad()) Py_RETURN_NONE;
    const float *bias = nullptr;
    if (n > 1 && args[1] != Py_None) {
        if (!plain_tensor(args[1])) Py_RETURN_NONE;
        const Tensor &b = THPVariable_Unpack(args[1]);
        if ((grad && b.requires_grad()) || !float_vector(b, device, p->rows)) Py_RETURN_NONE;
        bias = b.const_data_ptr<float>();
    }
    at::ScalarType out_type = x.scalar_type();
    if (n > 2 && args[2] != Py_None) {
        if (!THPDtype_Check(args[2])) Py_RETURN_NONE;
        out_type = reinterpret_cast<THPDtype *>(args[2])->scalar_type;
        if (dtype_code(out_type) < 0) Py_RETURN_NONE;
    }
    int64_t shape[3] = {x.size(0), x.dim() == 3 ? x.size(1) : p->rows, p->rows};
    try {
        return THPVariable_Wrap(product(*p->t2, p->rows, p->k, p->row_scale ? p->row_scale->const_data_ptr<float>() : nullptr, bias, rows,
                                        c10::IntArrayRef(shape, x.dim()), out_type, device, 2));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    END_HANDLE_TH_ERRORS
}

PyObject *product_new(PyTypeObject *type, PyObject *args, PyObject *) {
    HANDLE_TH_ERRORS
    PyObject *t2, *scale;
    long long rows, k;
    if (!PyArg_ParseTuple(args, "OLLO", &t2, &rows, &k, &scale)) return nullptr;
    TORCH_CHECK_VALUE(plain_tensor(t2) && (scale == Py_None || plain_tensor(scale)), "Product: expected tensors");
    const Tensor &w = THPVariable_Unpack(t2);
    TORCH_CHECK_VALUE(w.is_cuda() && w.scalar_type() == at::kByte && w.is_contiguous() && rows > 0 && k > 0 && w.numel() == t81b200_t2_bytes(rows, k),
                      "Product: t2 does not hold a rows x k matrix");
    if (scale != Py_None)
        TORCH_CHECK_VALUE(float_vector(THPVariable_Unpack(scale), w.device(), rows), "Product: row_scale must be float32 (rows,) on the weight's device");
    auto *self = reinterpret_cast<ProductObject *>(type->tp_alloc(type, 0));
    if (!self) return nullptr;
    self->call = product_call;
    self->t2 = new Tensor(w);
    self->row_scale = scale == Py_None ? nullptr : new Tensor(THPVariable_Unpack(scale));
    self->rows = rows;
    self->k = k;
    return reinterpret_cast<PyObject *>(self);
    END_HANDLE_TH_ERRORS
}

void product_dealloc(PyObject *o) {
    auto *self = reinterpret_cast<ProductObject *>(o);
    delete self->t2;
    delete self->row_scale;
    Py_TYPE(o)->tp_free(o);
}

PyTypeObject ProductType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- the training step of a Linear (t81/nn/linear.py:72-99 through t81/qat.py:12-57) ----

Tensor with_unit_columns(const Tensor &t) { return t.stride(1) == 1 && (t.size(0) < 2 || t.stride(0) >= t.size(1)) ? t : t.contiguous(); }

// Token-major rows as an operand of the gradient products.
Rows rows_of(const Tensor &t) {
    Rows r;
    r.data = t.const_data_ptr();
    r.dtype = dtype_code(t.scalar_type());
    r.tokens = t.size(0);
    r.ld = r.tokens > 1 ? t.stride(0) : t.size(1);
    return r;
}

// The same rows staged for TMA where they cannot be read in place; `keep` holds the copy.
Rows staged(const Rows &r, int64_t width, const c10::Device &device, Tensor &keep) {
    if (r.tokens == 0 || (r.dtype != T81B200_F32 && reinterpret_cast<uintptr_t>(r.data) % 16 == 0 && r.ld % 8 == 0)) return r;
    OnDevice on(device);
    keep = at::empty({(int64_t)t81b200_stage_rows_bytes(r.dtype, r.tokens, width)}, at::TensorOptions().dtype(at::kByte).device(device));
    check(t81b200_stage_rows(r.data, r.dtype, r.ld, r.tokens, width, keep.mutable_data_ptr(), stream_of(device)));
    Rows s = r;
    s.data = keep.const_data_ptr();
    s.ld = t81b200_stage_rows_ld(width);
    if (r.dtype == T81B200_F32) s.dtype = T81B200_BF16X3;
    return s;
}

Tensor weight_grad(const Rows &g, const Rows &x, const Tensor &w, const Tensor &scale) {
    const int64_t rows = w.size(0), cols = w.size(1);
    OnDevice on(w.device());
    Tensor out = at::empty({rows, cols}, w.options());
    const size_t need = t81b200_qat_weight_grad_workspace_bytes(g.data, g.dtype, g.ld, x.data, x.dtype, x.ld, x.tokens, rows, cols);
    Tensor ws;
    if (need) ws = at::empty({(int64_t)need}, w.options().dtype(at::kByte));
    check(t81b200_qat_weight_grad(g.data, g.dtype, g.ld, x.data, x.dtype, x.ld, x.tokens, rows, cols, w.const_data_ptr<float>(), rows > 1 ? w.stride(0) : cols,
                                  scale.const_data_ptr<float>(), out.mutable_data_ptr<float>(), need ? ws.mutable_data_ptr() : nullptr, need,
                                  stream_of(w.device())));
    return out;
}

struct QatLinear : public torch::autograd::Function<QatLinear> {
    using Context = torch::autograd::AutogradContext;

    // x: token-major rows; state: the layer's four floats, the scale updated by the caller; threshold in [0, 1]
    static Tensor forward(Context *ctx, const Tensor &x, const Tensor &weight, const std::optional<Tensor> &bias, const Tensor &state, double threshold) {
        const c10::Device device = weight.device();
        const int64_t rows = weight.size(0), cols = weight.size(1);
        OnDevice on(device);
        const Tensor w = with_unit_columns(weight);
        const bool grad_x = x.requires_grad();
        const auto bytes = w.options().dtype(at::kByte);
        Tensor t2 = at::empty({t81b200_t2_bytes(rows, cols)}, bytes), scales = at::empty({rows > cols ? rows : cols}, w.options()), t2_t;
        if (grad_x) t2_t = at::empty({t81b200_t2_bytes(cols, rows)}, bytes);
        check(t81b200_qat_quantize_t2(w.const_data_ptr<float>(), rows, cols, rows > 1 ? w.stride(0) : cols, (float)threshold, state.const_data_ptr<float>(),
                                      t2.mutable_data_ptr<uint8_t>(), grad_x ? t2_t.mutable_data_ptr<uint8_t>() : nullptr, scales.mutable_data_ptr<float>(),
                                      scales.numel(), stream_of(device)));
        std::optional<Tensor> b = bias;
        if (b) b = b->to(device, at::kFloat).contiguous();
        Rows r;
        TORCH_CHECK_VALUE(as_rows(x, cols, r), "t81.nn.Linear: input does not match in_features");
        Tensor y = product(t2, rows, cols, scales.const_data_ptr<float>(), float_ptr(b), r, {r.tokens, rows}, x.scalar_type(), device, 2);
        // the gradients use this step's scale, whatever later steps make of the layer's state
        ctx->save_for_backward({x, weight, scales.narrow(0, 0, 1)});
        ctx->saved_data["scales"] = scales;
        ctx->saved_data["t2_t"] = t2_t;
        ctx->saved_data["bias"] = bias ? bias->requires_grad() : false;
        ctx->saved_data["weight"] = weight.requires_grad();
        ctx->saved_data["threshold"] = threshold;
        return y;
    }

    static torch::autograd::variable_list backward(Context *ctx, torch::autograd::variable_list grads) {
        return as_python_error([&] { return gradients(ctx, grads); });
    }

    static torch::autograd::variable_list gradients(Context *ctx, const torch::autograd::variable_list &grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &weight = saved[1], &scale = saved[2];
        const int64_t rows = weight.size(0), cols = weight.size(1);
        // hooks on saved tensors may hand them back elsewhere and laid out otherwise
        const c10::Device device = grads[0].device();
        TORCH_CHECK_VALUE(saved[0].device() == device && weight.device() == device && scale.device() == device, "saved tensors of the training step are not on ", device);
        const Tensor x2 = with_unit_columns(saved[0]);
        if (at::GradMode::is_enabled() || !grads[0].has_storage() || grads[0].is_neg()) return recorded_gradients(ctx, grads[0], x2, weight, scale);
        const Tensor g = with_unit_columns(grads[0]);
        const Tensor scales = ctx->saved_data["scales"].toTensor(), t2_t = ctx->saved_data["t2_t"].toTensor();
        Tensor grad_x, grad_w, grad_b;
        const bool want_w = ctx->saved_data["weight"].toBool();
        Rows r = rows_of(g);
        Tensor keep;  // both products read one staged copy
        if (t2_t.defined() && want_w) r = staged(r, rows, weight.device(), keep);
        if (t2_t.defined()) {
            // every mantissa bit of a float32 gradient counts here: three planes
            grad_x = product(t2_t, cols, rows, scales.const_data_ptr<float>(), nullptr, r, {r.tokens, cols}, g.scalar_type(), weight.device(), 3);
        }
        if (want_w) grad_w = weight_grad(r, rows_of(x2), with_unit_columns(weight), scale);
        if (ctx->saved_data["bias"].toBool()) {
            OnDevice on(g.device());
            grad_b = at::empty({rows}, weight.options());
            check(t81b200_column_sums(g.const_data_ptr(), dtype_code(g.scalar_type()), g.size(0), rows, g.size(0) > 1 ? g.stride(0) : rows,
                                      grad_b.mutable_data_ptr<float>(), stream_of(g.device())));
        }
        return {grad_x, grad_w, grad_b, Tensor(), Tensor()};
    }

    // The same gradients in torch's operations: where they are differentiated again (create_graph) or the output's gradient is no
    // plain memory (a batch of them under vmap).  The weight enters through its surrogate, as in the PyTorch form of the step.
    static torch::autograd::variable_list recorded_gradients(Context *ctx, const Tensor &g, const Tensor &x, const Tensor &weight, const Tensor &scale) {
        const double threshold = ctx->saved_data["threshold"].toDouble();
        const Tensor ratio = weight.detach() / scale, slope = (ratio.abs() < 0.5).to(at::kFloat) * 2.0;
        Tensor grad_x, grad_w, grad_b;
        if (ctx->saved_data["t2_t"].toTensor().defined()) {
            const Tensor trits = at::logical_and(ratio >= threshold, ratio > 0).to(at::kFloat) - at::logical_and(ratio <= -threshold, ratio < 0).to(at::kFloat);
            const Tensor w = trits * scale + slope * (weight - weight.detach()).nan_to_num(0.0, 0.0, 0.0);
            grad_x = g.matmul(w.to(g.scalar_type()));
        }
        if (ctx->saved_data["weight"].toBool()) grad_w = g.to(at::kFloat).t().matmul(x.to(at::kFloat)) * slope;
        if (ctx->saved_data["bias"].toBool()) grad_b = g.sum(at::IntArrayRef{0});
        return {grad_x, grad_w, grad_b, Tensor(), Tensor()};
    }
};

std::optional<Tensor> optional_tensor(PyObject *o) {
    if (o == Py_None) return std::nullopt;
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor or None");
    return THPVariable_Unpack(o);
}
const Tensor &tensor_of(PyObject *o) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
    return THPVariable_Unpack(o);
}

// qat_linear(x, weight, bias, state, momentum, threshold): updates the running scale, then the forward above.
PyObject *qat_linear(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6) return PyErr_Format(PyExc_TypeError, "qat_linear takes 6 arguments");
    const Tensor x = tensor_of(args[0]), weight = tensor_of(args[1]), state = tensor_of(args[3]);
    const std::optional<Tensor> bias = optional_tensor(args[2]);
    const double momentum = PyFloat_AsDouble(args[4]), threshold = PyFloat_AsDouble(args[5]);
    if (PyErr_Occurred()) return nullptr;
    TORCH_CHECK_VALUE(weight.dim() == 2 && weight.scalar_type() == at::kFloat && weight.is_cuda() && x.device() == weight.device() && x.dim() >= 1 &&
                          x.size(-1) == weight.size(1) && float_vector(state, weight.device(), 4),
                      "qat_linear: x and weight do not match");
    return THPVariable_Wrap(as_python_error([&] {
        const Tensor w = with_unit_columns(weight.detach());
        {
            OnDevice on(w.device());
            check(t81b200_qat_update_scale(w.const_data_ptr(), T81B200_F32, w.size(0), w.size(1), w.size(0) > 1 ? w.stride(0) : w.size(1), (float)momentum,
                                           state.mutable_data_ptr<float>(), stream_of(w.device())));
        }
        // what the input needs on its way in and out is torch's to record; the node itself takes token-major rows
        Tensor rows = x.dim() == 2 ? x : x.reshape({-1, weight.size(1)});
        if (dtype_code(rows.scalar_type()) < 0) rows = rows.to(at::kFloat);
        const Tensor y = QatLinear::apply(with_unit_columns(rows), weight, bias, state, threshold);
        if (x.dim() == 2) return y;
        auto shape = x.sizes().vec();
        shape.back() = weight.size(0);
        return y.reshape(shape);
    }));
    END_HANDLE_TH_ERRORS
}

// linear_t2(t2, rows, x, k, row_scale, bias, out_dtype or None, fp32_planes) for 2-D x with unit column stride.
PyObject *linear_t2(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) return PyErr_Format(PyExc_TypeError, "linear_t2 takes 8 arguments");
    const Tensor &t2 = tensor_of(args[0]), &x = tensor_of(args[2]);
    const int64_t rows = PyLong_AsLongLong(args[1]), k = PyLong_AsLongLong(args[3]);
    const std::optional<Tensor> scale = optional_tensor(args[4]), bias = optional_tensor(args[5]);
    const int planes = (int)PyLong_AsLong(args[7]);
    if (PyErr_Occurred()) return nullptr;
    at::ScalarType out_type = x.scalar_type();
    if (args[6] != Py_None) {
        TORCH_CHECK_TYPE(THPDtype_Check(args[6]), "out_dtype must be a torch.dtype");
        out_type = reinterpret_cast<THPDtype *>(args[6])->scalar_type;
    }
    Rows r;
    TORCH_CHECK_VALUE(x.dim() == 2 && x.is_cuda() && x.device() == t2.device() && as_rows(x, k, r) && dtype_code(out_type) >= 0,
                      "linear_t2: x must be (tokens, K) float32, bfloat16 or float16 rows on the weight's device");
    TORCH_CHECK_VALUE(t2.numel() == t81b200_t2_bytes(rows, k) && (!scale || (float_vector(*scale, x.device(), scale->numel()) && scale->numel() >= rows)) &&
                          (!bias || float_vector(*bias, x.device(), rows)),
                      "linear_t2: weight, row_scale or bias do not match");
    try {
        return THPVariable_Wrap(product(t2, rows, k, float_ptr(scale), float_ptr(bias), r, {r.tokens, rows}, out_type, x.device(), planes));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    END_HANDLE_TH_ERRORS
}

PyObject *qat_weight_grad(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) return PyErr_Format(PyExc_TypeError, "qat_weight_grad takes 4 arguments");
    const Tensor &g = tensor_of(args[0]), &x = tensor_of(args[1]), &w = tensor_of(args[2]), &scale = tensor_of(args[3]);
    TORCH_CHECK_VALUE(w.dim() == 2 && g.dim() == 2 && x.dim() == 2 && w.scalar_type() == at::kFloat && w.is_cuda() && w.stride(1) == 1 &&
                          g.device() == w.device() && x.device() == w.device() && g.scalar_type() == x.scalar_type() && dtype_code(x.scalar_type()) >= 0 &&
                          g.size(0) == x.size(0) && g.size(1) == w.size(0) && x.size(1) == w.size(1) && float_vector(scale, w.device(), 1),
                      "qat_weight_grad: operands do not match");
    try {
        return THPVariable_Wrap(weight_grad(rows_of(with_unit_columns(g)), rows_of(with_unit_columns(x)), w, scale));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    END_HANDLE_TH_ERRORS
}

int64_t limbs_of(int64_t cols) { return (cols + 47) / 48; }

// quantize_pack(w, threshold, rule, out or None, row_scale_out or None) -> (packed, row_scale or None)
PyObject *quantize_pack(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5) return PyErr_Format(PyExc_TypeError, "quantize_pack takes 5 arguments");
    const Tensor *w = &tensor_of(args[0]);
    const double threshold = PyFloat_AsDouble(args[1]);
    const int rule = (int)PyLong_AsLong(args[2]);
    std::optional<Tensor> packed = optional_tensor(args[3]), scale = optional_tensor(args[4]);
    if (PyErr_Occurred()) return nullptr;
    TORCH_CHECK_VALUE(w->dim() == 2, "pack_dense_matrix expects a 2D array");
    TORCH_CHECK_VALUE(w->is_cuda(), "w must be a CUDA tensor (there is no CPU path)");
    const int dtype = dtype_code(w->scalar_type());
    TORCH_CHECK_VALUE(dtype >= 0, "w must be float32, bfloat16 or float16, got ", w->dtype());
    const c10::Device device = w->device();
    const int64_t rows = w->size(0), cols = w->size(1), kl = limbs_of(cols);
    OnDevice on(device);
    Tensor unit;
    if (w->numel() > 0 && (w->stride(1) != 1 || (rows > 1 && w->stride(0) < cols))) {
        unit = w->contiguous();
        w = &unit;
    }
    if (packed) {
        TORCH_CHECK_VALUE(packed->numel() == rows * kl * 16 && packed->scalar_type() == at::kByte && packed->is_contiguous() && packed->device() == device,
                          "packed output buffer has the wrong size");
    } else packed = at::empty({rows, kl, 16}, at::TensorOptions().dtype(at::kByte).device(device));
    if (rule == T81B200_RULE_ABSMEAN) {
        if (scale) {
            TORCH_CHECK_VALUE(float_vector(*scale, device, rows), "row_scale output must be float32 (rows,) on the weight's device");
        } else scale = at::empty({rows}, at::TensorOptions().dtype(at::kFloat).device(device));
    } else scale.reset();
    try {
        check(t81b200_quantize_pack(w->const_data_ptr(), dtype, rows, cols, rows > 1 ? w->stride(0) : (cols > 1 ? cols : 1), (float)threshold, rule,
                                    packed->mutable_data_ptr<uint8_t>(), scale ? scale->mutable_data_ptr<float>() : nullptr, stream_of(device)));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    PyObject *result = PyTuple_New(2);
    if (!result) return nullptr;
    PyTuple_SET_ITEM(result, 0, THPVariable_Wrap(*packed));
    PyTuple_SET_ITEM(result, 1, scale ? THPVariable_Wrap(*scale) : Py_NewRef(Py_None));
    return result;
    END_HANDLE_TH_ERRORS
}

// tensor_body(device_of, rows, cols): a (rows, cols) view of one element, the data-less body of a TernaryTensor.
PyObject *tensor_body(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 3) return PyErr_Format(PyExc_TypeError, "tensor_body takes 3 arguments");
    const Tensor &like = tensor_of(args[0]);
    const int64_t rows = PyLong_AsLongLong(args[1]), cols = PyLong_AsLongLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    at::AutoDispatchBelowADInplaceOrView below;
    return THPVariable_Wrap(at::empty({1}, at::TensorOptions().dtype(at::kFloat).device(like.device())).expand({rows, cols}));
    END_HANDLE_TH_ERRORS
}

// packed_to_tq(packed, rows, cols, format, row_scale or None) -> blocks
PyObject *packed_to_tq(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5) return PyErr_Format(PyExc_TypeError, "packed_to_tq takes 5 arguments");
    const Tensor packed = tensor_of(args[0]).contiguous();
    const int64_t rows = PyLong_AsLongLong(args[1]), cols = PyLong_AsLongLong(args[2]);
    const int format = (int)PyLong_AsLong(args[3]);
    std::optional<Tensor> scale = optional_tensor(args[4]);
    if (PyErr_Occurred()) return nullptr;
    const c10::Device device = packed.device();
    TORCH_CHECK_VALUE(packed.is_cuda(), "packed must be a CUDA tensor (there is no CPU path)");
    TORCH_CHECK_VALUE(rows >= 0 && cols >= 0 && packed.nbytes() >= (size_t)(rows * limbs_of(cols) * 16), "packed does not hold rows x ceil(cols/48) limbs");
    if (scale) {
        scale = scale->to(device, at::kFloat).contiguous();
        TORCH_CHECK_VALUE(scale->numel() >= rows, "row_scale must have one value per row");
    }
    OnDevice on(device);
    Tensor out = at::empty({rows, (cols + 255) / 256, format == T81B200_TQ2_0 ? 66 : 54}, at::TensorOptions().dtype(at::kByte).device(device));
    try {
        check(t81b200_packed_to_tq(static_cast<const uint8_t *>(packed.const_data_ptr()), float_ptr(scale), rows, cols, format, out.mutable_data_ptr<uint8_t>(),
                                   stream_of(device)));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// tq_to_packed(blocks, rows, cols, format) -> (packed, block_scales)
PyObject *tq_to_packed(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) return PyErr_Format(PyExc_TypeError, "tq_to_packed takes 4 arguments");
    const Tensor blocks = tensor_of(args[0]).contiguous();
    const int64_t rows = PyLong_AsLongLong(args[1]), cols = PyLong_AsLongLong(args[2]);
    const int format = (int)PyLong_AsLong(args[3]);
    if (PyErr_Occurred()) return nullptr;
    const c10::Device device = blocks.device();
    TORCH_CHECK_VALUE(blocks.is_cuda(), "blocks must be a CUDA tensor (there is no CPU path)");
    TORCH_CHECK_VALUE((int64_t)blocks.numel() == t81b200_tq_bytes(format, rows, cols) && blocks.element_size() == 1, "block payload size does not match (rows, cols)");
    OnDevice on(device);
    const auto options = at::TensorOptions().device(device);
    Tensor packed = at::empty({rows, limbs_of(cols), 16}, options.dtype(at::kByte)), scales = at::empty({rows, (cols + 255) / 256}, options.dtype(at::kFloat));
    try {
        check(t81b200_tq_to_packed(static_cast<const uint8_t *>(blocks.const_data_ptr()), rows, cols, format, packed.mutable_data_ptr<uint8_t>(),
                                   scales.mutable_data_ptr<float>(), stream_of(device)));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    PyObject *result = PyTuple_New(2);
    if (!result) return nullptr;
    PyTuple_SET_ITEM(result, 0, THPVariable_Wrap(packed));
    PyTuple_SET_ITEM(result, 1, THPVariable_Wrap(scales));
    return result;
    END_HANDLE_TH_ERRORS
}

// gemm_trit(packed, B, C, layout, M, N, K, row_scale or None, bias or None, alpha, beta): operands checked by the caller.
PyObject *gemm_trit(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 11) return PyErr_Format(PyExc_TypeError, "gemm_trit takes 11 arguments");
    const Tensor &packed = tensor_of(args[0]), &B = tensor_of(args[1]), &C = tensor_of(args[2]);
    const int layout = (int)PyLong_AsLong(args[3]);
    const int64_t M = PyLong_AsLongLong(args[4]), N = PyLong_AsLongLong(args[5]), K = PyLong_AsLongLong(args[6]);
    const std::optional<Tensor> scale = optional_tensor(args[7]), bias = optional_tensor(args[8]);
    const double alpha = PyFloat_AsDouble(args[9]), beta = PyFloat_AsDouble(args[10]);
    if (PyErr_Occurred()) return nullptr;
    const int b_dtype = dtype_code(B.scalar_type()), c_dtype = dtype_code(C.scalar_type());
    const c10::Device device = B.device();
    const int64_t ldb = B.size(0) > 1 ? B.stride(0) : (B.size(1) > 1 ? B.size(1) : 1), ldc = C.size(0) > 1 ? C.stride(0) : (C.size(1) > 1 ? C.size(1) : 1);
    OnDevice on(device);
    // 16-bit token-major rows on 16-byte boundaries are read in place, and up to 16 rows always are; the rest is staged
    // (bf16 rows off those boundaries too, where the problem is large enough)
    size_t need = 0;
    const bool token_major = layout == T81B200_LAYOUT_NK;
    const bool in_place = token_major && (N <= 16 || (b_dtype != T81B200_F32 && reinterpret_cast<uintptr_t>(B.const_data_ptr()) % 16 == 0 && ldb % 8 == 0));
    if (!in_place) {
        need = t81b200_gemm_trit_workspace_bytes(b_dtype, layout, c_dtype, M, N, K);
        if (need == 0 && token_major && (double)M * N * K >= 1.6e7) need = (size_t)N * ((K + 7) / 8 * 8) * 2;
    }
    Tensor ws;
    if (need) ws = at::empty({(int64_t)need}, at::TensorOptions().dtype(at::kByte).device(device));
    try {
        check(t81b200_gemm_trit(static_cast<const uint8_t *>(packed.const_data_ptr()), float_ptr(scale), B.const_data_ptr(), b_dtype, layout, ldb,
                                float_ptr(bias), C.mutable_data_ptr(), c_dtype, ldc, M, N, K, (float)alpha, (float)beta,
                                need ? ws.mutable_data_ptr() : nullptr, need, stream_of(device)));
    } catch (const LibraryError &e) {
        return raise_library_error(e.code);
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"quantize_pack", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(quantize_pack)), METH_FASTCALL, nullptr},
    {"tensor_body", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tensor_body)), METH_FASTCALL, nullptr},
    {"packed_to_tq", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(packed_to_tq)), METH_FASTCALL, nullptr},
    {"tq_to_packed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tq_to_packed)), METH_FASTCALL, nullptr},
    {"gemm_trit", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm_trit)), METH_FASTCALL, nullptr},
    {"qat_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(qat_linear)), METH_FASTCALL, nullptr},
    {"linear_t2", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_t2)), METH_FASTCALL, nullptr},
    {"qat_weight_grad", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(qat_weight_grad)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_t81_torch", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__t81_torch() {
    ProductType.tp_name = "t81lib_b200._t81_torch.Product";
    ProductType.tp_basicsize = sizeof(ProductObject);
    ProductType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    ProductType.tp_new = product_new;
    ProductType.tp_dealloc = product_dealloc;
    ProductType.tp_call = PyVectorcall_Call;
    ProductType.tp_vectorcall_offset = offsetof(ProductObject, call);
    if (PyType_Ready(&ProductType) < 0) return nullptr;
    PyObject *m = PyModule_Create(&module);
    if (!m) return nullptr;
    Py_INCREF(&ProductType);
    PyModule_AddObject(m, "Product", reinterpret_cast<PyObject *>(&ProductType));
    return m;
}
