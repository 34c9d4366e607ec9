// The calls of a decode loop that are bound by the host (ops.mmv, ops.linear, ops.draft_logits) in native code: the same checks, the
// same allocations and launches as the Python functions, whose attribute reads, ctypes structures and device guard took 14 us of
// an 8192 x 2048 product's 23 (8 are the kernel's). Each function returns None for a call that it does not take as it is - another
// tensor type, a torch-function or dispatch mode, a functorch wrapper, another current device, or arguments that the Python function would refuse or copy -
// and the Python function goes on from there, so refusals and their messages are its own. Nothing is kept between calls.
#include "../../include/bf16n_c.h"

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <algorithm>
#include <vector>

namespace {

PyTypeObject * g_weight, * g_meta; // ops.Weight, ops.Meta
PyObject * s_plane, * s_aux, * s_meta, * s_marks, * s_marks_at;
const char * const META_FIELDS[10] = {"format", "K", "rows", "R", "chunk_major", "frag_order", "off_a", "off_b", "off_c", "off_d"};
PyObject * s_fields[10];

struct Ref { // an owned reference
    PyObject * p;
    explicit Ref(PyObject * o) : p(o) {}
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref &) = delete;
    Ref & operator=(const Ref &) = delete;
};

// an ordinary CUDA tensor, which the functions below may take apart
bool plain(PyObject * o) {
    if (!THPVariable_CheckExact(o)) { return false; }
    const at::Tensor & t = THPVariable_Unpack(o);
    constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                           c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative});
    return t.defined() && t.is_cuda() && t.layout() == c10::kStrided && t.has_storage() && !t.key_set().has_any(wrapped);
}
bool modes_active() {
    return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() || torch::jit::tracer::isTracing();
}

struct Matrix { bf16n_weight c; const void * marks; c10::Device device{c10::kCPU}; };

// ops.Weight.c() and marks_ptr(); false: not an ordinary weight on the current device, or one that c() refuses
bool matrix_of(PyObject * w, Matrix & m) {
    if (Py_TYPE(w) != g_weight) { return false; }
    Ref plane(PyObject_GetAttr(w, s_plane)), aux(PyObject_GetAttr(w, s_aux)), meta(PyObject_GetAttr(w, s_meta)), marks(PyObject_GetAttr(w, s_marks));
    if (!plane.p || !aux.p || !meta.p || !marks.p) { PyErr_Clear(); return false; }
    if (Py_TYPE(meta.p) != g_meta || !plain(plane.p) || !plain(aux.p)) { return false; }
    long long v[10];
    for (int i = 0; i < 10; i++) {
        Ref f(PyObject_GetAttr(meta.p, s_fields[i]));
        if (!f.p) { PyErr_Clear(); return false; }
        v[i] = PyLong_AsLongLong(f.p);
        if (v[i] == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    }
    const at::Tensor & p = THPVariable_Unpack(plane.p), & a = THPVariable_Unpack(aux.p);
    if (p.scalar_type() != at::kByte || a.scalar_type() != at::kByte || !p.is_contiguous() || !a.is_contiguous() || p.device() != a.device()) { return false; }
    if (p.numel() != v[2] * v[1] || std::max(std::max(v[6], v[7]), std::max(v[8], v[9])) >= a.numel()) { return false; }
    if (p.device().index() != c10::cuda::current_device()) { return false; }
    m.c = {(const uint8_t *) p.const_data_ptr(), (const uint8_t *) a.const_data_ptr(), (int32_t) v[0], (int32_t) v[3], v[1], v[2], (int32_t) (v[4] != 0),
           (int32_t) (v[5] != 0), (uint64_t) v[6], (uint64_t) v[7], (uint64_t) v[8], (uint64_t) v[9]};
    m.device = p.device();
    m.marks = nullptr;
    if (marks.p != Py_None) {
        if (!plain(marks.p)) { return false; }
        const at::Tensor & k = THPVariable_Unpack(marks.p);
        Ref at(PyObject_GetAttr(w, s_marks_at));
        if (!at.p) { PyErr_Clear(); return false; }
        if (at.p != Py_None) { // aux was written since they were made: the Python function makes them again
            const long long made = PyLong_AsLongLong(at.p);
            if (made == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
            if (a.is_inference() || (long long) a._version() != made) { return false; }
        }
        const bool whole = k.is_contiguous() && (size_t) k.numel() * k.element_size() == bf16n_marks_bytes(&m.c);
        if (k.device() == m.device && whole && (uintptr_t) k.const_data_ptr() % 2 == 0) { m.marks = k.const_data_ptr(); }
    }
    return true;
}

// a failed call as the Python layer's check() raises it
struct Refused { int rc; };
void ok(int rc) { if (rc != BF16N_OK) { throw Refused{rc}; } }

template <typename F>
PyObject * guarded(F && f) {
    HANDLE_TH_ERRORS
    try {
        return f();
    } catch (const Refused & e) {
        PyErr_SetString(e.rc == BF16N_EINVAL ? PyExc_ValueError : PyExc_RuntimeError, bf16n_last_error());
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

struct NoGil { // as ctypes releases it for the time of a call
    PyThreadState * s = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(s); }
};

void * stream_of(const c10::Device & d) { return (void *) c10::cuda::getCurrentCUDAStream(d.index()).stream(); }

bool aligned16(const at::Tensor & x, int64_t stride0) { return (uintptr_t) x.const_data_ptr() % 16 == 0 && (stride0 * x.element_size()) % 16 == 0; }

// x [T, K] (rows `stride0` elements apart) through the decode GEMV into y [T, rows]
void gemv(const Matrix & m, const at::Tensor & x, int64_t T, int64_t stride0, at::Tensor & y, bool multi_col) {
    bf16n_mmv_args a = {};
    const bool y_bf16 = y.scalar_type() == at::kBFloat16;
    a.x = x.const_data_ptr(); a.x_bf16 = x.scalar_type() == at::kBFloat16;
    a.y = y.mutable_data_ptr(); a.y_bf16 = y_bf16;
    a.ncols = (int32_t) T; a.n_used = 1; a.x_per_slot = 1;
    a.x_tok = stride0 * x.element_size(); a.y_tok = m.c.rows * (y_bf16 ? 2 : 4);
    a.rows_per_matrix = a.nrows = m.c.rows;
    ok(bf16n_mmv_marked(&m.c, m.marks, &a, stream_of(m.device), multi_col));
}

// mmv(x, w, out_bf16, multi_col): dense, a new output
PyObject * call_mmv(PyObject *, PyObject * const * args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Matrix m;
        if (n != 4 || !plain(args[0]) || modes_active() || !matrix_of(args[1], m)) { Py_RETURN_NONE; }
        const at::Tensor & x = THPVariable_Unpack(args[0]);
        const bool out_bf16 = args[2] == Py_True, multi_col = args[3] == Py_True;
        if (x.dim() != 2 || x.size(0) == 0 || x.size(1) != m.c.K || x.stride(1) != 1 || x.device() != m.device) { Py_RETURN_NONE; }
        if (!(x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat) || !aligned16(x, x.stride(0))) { Py_RETURN_NONE; }
        at::Tensor y;
        {
            NoGil free;
            y = at::empty({x.size(0), m.c.rows}, x.options().dtype(out_bf16 ? at::kBFloat16 : at::kFloat).requires_grad(false));
            gemv(m, x, x.size(0), x.stride(0), y, multi_col);
        }
        return THPVariable_Wrap(std::move(y));
    });
}

// linear(x, w, bias, most_tokens, chunk_bytes)
PyObject * call_linear(PyObject *, PyObject * const * args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Matrix m;
        if (n != 5 || !plain(args[0]) || (args[2] != Py_None && !plain(args[2])) || modes_active() || !matrix_of(args[1], m)) { Py_RETURN_NONE; }
        const at::Tensor & x = THPVariable_Unpack(args[0]);
        if (x.scalar_type() != at::kBFloat16 || x.dim() < 2 || x.size(-1) != m.c.K || !x.is_contiguous() || x.device() != m.device || x.numel() == 0) { Py_RETURN_NONE; }
        const int64_t K = m.c.K, rows = m.c.rows, T = x.numel() / K, most = PyLong_AsLongLong(args[3]), chunk_bytes = PyLong_AsLongLong(args[4]);
        if (T <= most && !aligned16(x, K)) { Py_RETURN_NONE; }
        at::Tensor y;
        {
            NoGil free;
            const auto options = x.options().requires_grad(false);
            if (T <= most) {
                y = at::empty({T, rows}, args[2] == Py_None ? options : options.dtype(at::kFloat));
                gemv(m, x, T, K, y, true);
                if (args[2] != Py_None) { y = y.add_(THPVariable_Unpack(args[2])).to(at::kBFloat16); }
            } else {
                const at::Tensor x2 = x.dim() == 2 ? x : x.reshape({T, K});
                y = at::empty({T, rows}, options);
                const int64_t unit = m.c.format == BF16N_FMT_NIBBLE ? 1 : std::max(m.c.R, 1);
                const int64_t chunk = std::min(std::max(chunk_bytes / (K * 2) / unit * unit, unit), rows);
                for (int64_t r0 = 0; r0 < rows; r0 += chunk) {
                    const int64_t nr = std::min(chunk, rows - r0);
                    at::Tensor wc = at::empty({nr, K}, options);
                    ok(bf16n_dequant_marked(&m.c, m.marks, r0, nr, (uint16_t *) wc.mutable_data_ptr(), stream_of(m.device)));
                    at::Tensor ys = y.narrow(1, r0, nr);
                    if (ys.is_contiguous()) { at::mm_out(ys, x2, wc.t()); } else { ys.copy_(at::matmul(x2, wc.t())); }
                    if (args[2] != Py_None) { ys.add_(THPVariable_Unpack(args[2]).narrow(0, r0, nr)); }
                }
            }
            if (x.dim() != 2) {
                std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
                shape.back() = rows;
                y = y.view(shape);
            }
        }
        return THPVariable_Wrap(std::move(y));
    });
}

// draft_logits(h, w, bits, q, s, candidates, vocab): the fused step, for an h without derivatives
PyObject * call_draft(PyObject *, PyObject * const * args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Matrix m;
        if (n != 7 || !plain(args[0]) || !plain(args[3]) || !plain(args[4]) || modes_active() || !matrix_of(args[1], m)) { Py_RETURN_NONE; }
        const at::Tensor & h = THPVariable_Unpack(args[0]), & q = THPVariable_Unpack(args[3]), & s = THPVariable_Unpack(args[4]);
        const int64_t bits = PyLong_AsLongLong(args[2]), cands = PyLong_AsLongLong(args[5]), vocab = PyLong_AsLongLong(args[6]);
        if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
        if (h.dim() != 2 || h.size(0) == 0 || h.scalar_type() != at::kBFloat16 || !h.is_contiguous() || h.device() != m.device || h.requires_grad() ||
            h._fw_grad(0).defined() || (uintptr_t) h.const_data_ptr() % 16) { Py_RETURN_NONE; }
        const int64_t T = h.size(0), K = h.size(1);
        if (K != m.c.K || (bits != 2 && bits != 4) || q.dim() != 2 || s.dim() != 2) { Py_RETURN_NONE; }
        const int64_t rows = q.size(0);
        if (q.scalar_type() != at::kByte || !q.is_contiguous() || q.size(1) != K * bits / 8 || q.device() != m.device) { Py_RETURN_NONE; }
        if (s.scalar_type() != at::kFloat || !s.is_contiguous() || s.size(0) != rows || s.size(1) != K / 128 || s.device() != m.device) { Py_RETURN_NONE; }
        if (rows > std::min(m.c.rows, vocab)) { Py_RETURN_NONE; }
        at::Tensor out;
        {
            NoGil free;
            const auto f32 = h.options().dtype(at::kFloat).requires_grad(false);
            at::Tensor scores = at::empty({T, rows}, f32);
            void * st = stream_of(m.device);
            ok((bits == 2 ? bf16n_int2_gemv : bf16n_int4_gemv)(h.const_data_ptr(), (int) T, (const uint8_t *) q.const_data_ptr(), (const float *) s.const_data_ptr(),
                                                                rows, (int) K, (float *) scores.mutable_data_ptr(), st));
            at::Tensor cand = at::empty({T, cands}, f32.dtype(at::kInt)), cand_rows = at::empty({T * cands, K}, f32.dtype(at::kBFloat16));
            out = at::empty({T, vocab}, f32);
            ok(bf16n_draft_logits_marked((const float *) scores.const_data_ptr(), (int) T, rows, (int) cands, &m.c, m.marks, h.const_data_ptr(),
                                         (int32_t *) cand.mutable_data_ptr(), cand_rows.mutable_data_ptr(), (float *) out.mutable_data_ptr(), vocab, st));
        }
        return THPVariable_Wrap(std::move(out));
    });
}

// register(Weight, Meta): the classes whose instances are taken
PyObject * call_register(PyObject *, PyObject * const * args, Py_ssize_t n) {
    if (n != 2 || !PyType_Check(args[0]) || !PyType_Check(args[1])) { PyErr_SetString(PyExc_TypeError, "register(Weight, Meta)"); return nullptr; }
    Py_INCREF(args[0]); Py_INCREF(args[1]);
    g_weight = (PyTypeObject *) args[0];
    g_meta = (PyTypeObject *) args[1];
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"register", (PyCFunction) (void (*)(void)) call_register, METH_FASTCALL, nullptr},
    {"mmv", (PyCFunction) (void (*)(void)) call_mmv, METH_FASTCALL, nullptr},
    {"linear", (PyCFunction) (void (*)(void)) call_linear, METH_FASTCALL, nullptr},
    {"draft_logits", (PyCFunction) (void (*)(void)) call_draft, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__calls(void) {
    s_plane = PyUnicode_InternFromString("plane");
    s_aux = PyUnicode_InternFromString("aux");
    s_meta = PyUnicode_InternFromString("meta");
    s_marks = PyUnicode_InternFromString("marks");
    s_marks_at = PyUnicode_InternFromString("marks_at");
    for (int i = 0; i < 10; i++) { s_fields[i] = PyUnicode_InternFromString(META_FIELDS[i]); }
    return PyModule_Create(&module);
}
