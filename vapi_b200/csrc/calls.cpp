// The calls that a step of a few tokens makes most often, from Python's arguments to the launch in one piece: checks, outputs and the
// call of the kernel's C function.  Such a step (a prompt of a line: 65 products, 97 launches) is bound by what its launches cost the
// host, and of a product's 14 us there only about 3 are the launch; checking its operands one by one in Python, allocating its
// outputs through the Python binding and converting two dozen arguments through ctypes are the rest.
//
// A function here answers NotImplemented for anything but what the kernels take as it is (other types, layouts, devices or
// tensor classes): its caller in ops then goes through the same steps in Python, which name what is wrong.  A negative number is the C
// function's error code.  Once the C function has been called there is no way back to Python's steps, which would add to the stream, or move
// a state on, a second time: what goes wrong from there on is an error.  The C functions are given by address, so this library is linked
// with none of the kernels' ones.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>

namespace {

struct Bad {};                              // not for this file: NotImplemented

const at::Tensor* tensor(PyObject* o) {     // None: null
    if (o == Py_None) return nullptr;
    if (!THPVariable_CheckExact(o)) throw Bad{};
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_conj() || t.is_neg()) throw Bad{};
    return &t;
}
const at::Tensor& need(PyObject* o, at::ScalarType type, int64_t dim) {
    const at::Tensor* t = tensor(o);
    if (!t || t->scalar_type() != type || t->dim() != dim || !t->is_contiguous()) throw Bad{};
    return *t;
}
// a vector of floats, as many as the kernel reads or more (`most`: no more than that), or none
const float* floats(PyObject* o, int64_t least, int64_t most = INT64_MAX) {
    const at::Tensor* t = tensor(o);
    if (!t) return nullptr;
    if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() < least || t->numel() > most) throw Bad{};
    return static_cast<const float*>(t->data_ptr());
}
const int* ints(PyObject* o, int64_t least) {
    const at::Tensor* t = tensor(o);
    if (!t || t->scalar_type() != at::kInt || !t->is_contiguous() || t->numel() < least) throw Bad{};
    return static_cast<const int*>(t->data_ptr());
}
void* address(PyObject* o) {                // None: null
    if (o == Py_None) return nullptr;
    void* p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) { PyErr_Clear(); throw Bad{}; }
    return p;
}
int integer(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if ((v == -1 && PyErr_Occurred()) || v > 0x7fffffffL || v < -0x7fffffffL) { PyErr_Clear(); throw Bad{}; }
    return (int)v;
}
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); throw Bad{}; }
    return (float)v;
}
int size32(int64_t v) {
    if (v > 0x7fffffffLL) throw Bad{};
    return (int)v;
}
PyObject* wrap(const at::Tensor& t) {       // (null: a Python error)
    if (t.defined()) return THPVariable_Wrap(t);
    Py_RETURN_NONE;
}

// The interpreter's lock is given up while one of these lives, and taken again however its block is left.
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};

// body(called): sets `called` before it calls the C function
template <typename F>
PyObject* guarded(Py_ssize_t given, Py_ssize_t wanted, F&& body) {
    if (given != wanted) {
        PyErr_Format(PyExc_TypeError, "%zd arguments instead of %zd", given, wanted);
        return nullptr;
    }
    bool called = false;
    const char* what = "an unknown exception";
    std::string text;
    try {
        return body(called);
    } catch (const Bad&) {
    } catch (const std::exception& e) {     // (what torch objects to, the same calls in Python say)
        text = e.what();
        what = text.c_str();
    } catch (...) {
    }
    if (called) {
        if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "a kernel's launch ended with an exception: %s", what);
        return nullptr;
    }
    PyErr_Clear();
    Py_RETURN_NOTIMPLEMENTED;
}

typedef int (*PlanFn)(int, int, int, int, int*, int*, int*);
typedef int (*ProductFn)(const void*, int, int, int, int, const void*, const float*, int, float, int, void*, float*, long long, const float*,
                         float*, float*, const float*, void*, int*, void*, const float*, int);
enum { EPI_BF16 = 0, EPI_SWIGLU = 1, EPI_RESID = 2, EPI_F32 = 3 };

// product(fn, plan, which of the plan's answers is the partial sums of squares, weight, act, xw, ss_in, eps, epilogue, bias, resid,
//         next_weight, status, xielu, glu, stream): ops._fused_product
PyObject* product(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 16, [&](bool& called) -> PyObject* {
        const auto fn = reinterpret_cast<ProductFn>(address(a[0]));
        const auto plan = reinterpret_cast<PlanFn>(address(a[1]));
        const int answer = integer(a[2]), epi = integer(a[8]);
        if (!fn || !plan || answer < 0 || answer > 2 || epi < EPI_BF16 || epi > EPI_F32) throw Bad{};
        const at::Tensor& w = need(a[3], at::kBFloat16, 2);
        const bool norm = a[4] == Py_None;
        const at::Tensor& x = need(norm ? a[5] : a[4], at::kBFloat16, 2);
        const int N = size32(w.size(0)), K = size32(w.size(1)), M = size32(x.size(0));
        if (x.size(1) != K) throw Bad{};
        const float* ss = nullptr;
        int parts_in = 0;
        if (norm) {
            const at::Tensor& s = need(a[6], at::kFloat, 2);
            if (s.size(1) != M) throw Bad{};
            ss = static_cast<const float*>(s.data_ptr());
            parts_in = size32(s.size(0));
        } else if (a[6] != Py_None) {
            throw Bad{};
        }
        const float* bias = floats(a[9], N, N);
        const float* next_w = floats(a[11], N);
        const float* xielu = floats(a[13], 2);
        float* resid = nullptr;
        at::Tensor out, sums, weighted;
        const auto options = w.options();
        long long stride = N;
        if (epi == EPI_RESID) {
            const at::Tensor& r = need(a[10], at::kFloat, 2);
            if (r.size(0) != M || r.size(1) != N) throw Bad{};
            resid = static_cast<float*>(r.data_ptr());
            if (next_w) {
                int o[3] = {0, 0, 0};
                plan(N, K, M, epi, &o[0], &o[1], &o[2]);
                sums = at::empty({o[answer], M}, options.dtype(at::kFloat));
                weighted = at::empty({M, N}, options);
            }
        } else {
            if (a[10] != Py_None) throw Bad{};
            if (epi == EPI_SWIGLU) stride = N / 2;
            out = at::empty({M, stride}, epi == EPI_F32 ? options.dtype(at::kFloat) : options);
        }
        void* o = out.defined() ? out.data_ptr() : nullptr;
        float* so = sums.defined() ? static_cast<float*>(sums.data_ptr()) : nullptr;
        void* wo = weighted.defined() ? weighted.data_ptr() : nullptr;
        const float eps = real(a[7]);
        int* status = static_cast<int*>(address(a[12]));
        void* stream = address(a[15]);
        const int glu = integer(a[14]);
        int rc;
        called = true;
        {
            Unlocked unlocked;
            rc = fn(w.data_ptr(), N, K, M, norm ? 1 : 0, x.data_ptr(), ss, parts_in, eps, epi, epi == EPI_F32 ? nullptr : o,
                    epi == EPI_F32 ? static_cast<float*>(o) : nullptr, stride, bias, resid, so, next_w, wo, status, stream, xielu, glu);
        }
        if (rc != 0) return PyLong_FromLong(rc);
        if (epi != EPI_RESID) return wrap(out);
        PyObject* first = wrap(sums);
        PyObject* second = first ? wrap(weighted) : nullptr;
        PyObject* pair = second ? PyTuple_Pack(2, first, second) : nullptr;
        Py_XDECREF(first);
        Py_XDECREF(second);
        return pair;
    });
}

typedef int (*ShortconvFn)(const void*, int, const float*, const float*, const float*, void*, long long, const int*, const int*, const int*,
                           const int*, void*, int, int, int, int, int, int*, void*);

// shortconv(fn, h3, in_bias, taps, conv_bias, state, state_slots, tok_seq, cu_q, positions, status, stream): ops.shortconv in bfloat16
PyObject* shortconv(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 12, [&](bool& called) -> PyObject* {
        const auto fn = reinterpret_cast<ShortconvFn>(address(a[0]));
        const at::Tensor& h3 = need(a[1], at::kBFloat16, 2);
        const at::Tensor& taps = need(a[3], at::kFloat, 2);
        const int n = size32(h3.size(0)), H = size32(h3.size(1) / 3), L = size32(taps.size(0));
        if (!fn || h3.size(1) != 3LL * H || taps.size(1) != H) throw Bad{};
        const at::Tensor* state = tensor(a[5]);
        long long slot_stride = 0;
        int slots = 0;
        if (L > 1) {
            if (!state || state->scalar_type() != at::kBFloat16 || state->dim() != 3 || state->size(1) != L - 1 || state->size(2) != H ||
                state->stride(2) != 1 || state->stride(1) != H) throw Bad{};
            slot_stride = state->stride(0);
            slots = size32(state->size(0));
        }
        const at::Tensor* cu = tensor(a[8]);
        if (!cu || cu->scalar_type() != at::kInt || !cu->is_contiguous()) throw Bad{};
        const int seqs = size32(cu->numel() - 1);
        const float *in_bias = floats(a[2], 3LL * H), *conv_bias = floats(a[4], H);
        const int *state_slots = ints(a[6], seqs), *tok_seq = ints(a[7], n), *positions = ints(a[9], n);
        int* status = static_cast<int*>(address(a[10]));
        void* stream = address(a[11]);
        at::Tensor out = at::empty({n, H}, h3.options());
        int rc;
        called = true;
        {
            Unlocked unlocked;
            rc = fn(h3.data_ptr(), 1, in_bias, static_cast<const float*>(taps.data_ptr()), conv_bias, L > 1 ? state->data_ptr() : nullptr,
                    slot_stride, state_slots, tok_seq, static_cast<const int*>(cu->data_ptr()), positions, out.data_ptr(), n, seqs, H, L,
                    slots, status, stream);
        }
        return rc != 0 ? PyLong_FromLong(rc) : wrap(out);
    });
}

PyMethodDef methods[] = {
    {"product", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(product)), METH_FASTCALL, "a fused product of a few rows"},
    {"shortconv", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(shortconv)), METH_FASTCALL, "the gated short convolution"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "vapi_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_vapi_calls() { return PyModule_Create(&module); }
