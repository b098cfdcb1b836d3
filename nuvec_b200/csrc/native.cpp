// The host path of the Python operators: arrays and the marshalling of the usual calls, in C.
//
// Every operator of ops.py first offers its arguments to the function of the same name here.  If they are of the usual
// form -- arrays of one device, matching shapes and types -- the result is allocated, the C ABI is called and the result
// returned.  Anything else (an error to report, a promotion, a broadcast) is answered with None and nothing done; ops.py
// then takes its own path, which checks everything and words the errors.  So this file decides nothing: it only makes
// the common call cheap.  A call through ctypes with its shape arithmetic in Python cost 8-12 us, more than most decode
// products take on the GPU; the same call from here costs about 0.5 us plus the launch.
//
// The library's functions are bound by address (ops.py's ctypes handle), so this module links against nothing.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstddef>
#include <cstdint>

#include "../../include/nuvec_cuda.h"

namespace {

// ── the library ─────────────────────────────────────────────────────────────────────────
#define NVC_BOUND(X)                                                                                                             \
    X(nvc_alloc) X(nvc_free) X(nvc_quantize) X(nvc_dequantize) X(nvc_quantized_matmul) X(nvc_gather_qmm) X(nvc_moe_route)        \
    X(nvc_weighted_sum) X(nvc_expert_bias_add) X(nvc_moe_sort) X(nvc_take_rows) X(nvc_quantized_embedding) X(nvc_qqmm)           \
    X(nvc_qqmm_prepared) X(nvc_quantized_attention) X(nvc_rms_norm) X(nvc_add_rms_norm) X(nvc_swiglu) X(nvc_swiglu_oai)          \
    X(nvc_sorted_offsets)
#define NVC_DECLARE(name) decltype(&::name) name = nullptr;
struct Library {
    NVC_BOUND(NVC_DECLARE)
} L;
#undef NVC_DECLARE

// ── arrays ──────────────────────────────────────────────────────────────────────────────
struct DeviceObject {
    PyObject_HEAD
    nvc_device *handle;  // nullptr once closed
};
struct ArrayObject {
    PyObject_HEAD
    PyObject *dev, *shape, *base;  // base: the array whose memory this one looks at, or nullptr
    int dtype;
    Py_ssize_t offset;  // from the base's first byte
    char *data;
    bool owns;
};
PyTypeObject DeviceType = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyTypeObject ArrayType = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyTypeObject *array_class = nullptr;      // ops.Array
PyObject *quantized_class = nullptr;      // ops.Quantized
PyObject *modes[4] = {};                  // the members of ops.QuantMode by code
PyObject *s_weight, *s_scales, *s_biases, *s_quant, *s_global, *s_mode, *s_group, *s_bits, *s_ptr, *s_value;

bool is_array(PyObject *o) { return PyObject_TypeCheck(o, &ArrayType); }
ArrayObject *arr(PyObject *o) { return reinterpret_cast<ArrayObject *>(o); }
nvc_device *handle_of(const ArrayObject *a) { return reinterpret_cast<DeviceObject *>(a->dev)->handle; }
Py_ssize_t rank(const ArrayObject *a) { return PyTuple_GET_SIZE(a->shape); }
int64_t dim(const ArrayObject *a, Py_ssize_t i) { return PyLong_AsLongLong(PyTuple_GET_ITEM(a->shape, i < 0 ? i + rank(a) : i)); }
int64_t size_of(const ArrayObject *a) {
    int64_t n = 1;
    for (Py_ssize_t i = 0; i < rank(a); i++) n *= dim(a, i);
    return n;
}
int item_size(int dtype) { return dtype == NVC_U8 ? 1 : dtype == NVC_F16 || dtype == NVC_BF16 ? 2 : dtype == NVC_U32 || dtype == NVC_I32 || dtype == NVC_F32 ? 4 : 0; }
bool is_float(int dtype) { return dtype == NVC_F16 || dtype == NVC_BF16 || dtype == NVC_F32; }
bool same_shape(const ArrayObject *a, const ArrayObject *b) {
    if (rank(a) != rank(b)) return false;
    for (Py_ssize_t i = 0; i < rank(a); i++)
        if (dim(a, i) != dim(b, i)) return false;
    return true;
}

// A reference that is dropped at the end of the scope.
struct Ref {
    PyObject *o;
    explicit Ref(PyObject *p = nullptr) : o(p) {}
    ~Ref() { Py_XDECREF(o); }
    Ref(const Ref &) = delete;
    Ref &operator=(const Ref &) = delete;
    PyObject *release() {
        PyObject *p = o;
        o = nullptr;
        return p;
    }
    explicit operator bool() const { return o != nullptr; }
    ArrayObject *array() const { return arr(o); }
};

// Not the usual form: ops.py takes the call (whatever went wrong here, it finds again and words).
PyObject *decline() {
    PyErr_Clear();
    Py_RETURN_NONE;
}

PyObject *view_of(PyTypeObject *type, PyObject *dev, PyObject *shape /*stolen*/, int dtype, PyObject *base, Py_ssize_t offset, char *base_data) {
    ArrayObject *a = reinterpret_cast<ArrayObject *>(type->tp_alloc(type, 0));
    if (!a) {
        Py_DECREF(shape);
        return nullptr;
    }
    a->dev = Py_NewRef(dev);
    a->shape = shape;
    a->base = Py_NewRef(base);
    a->dtype = dtype;
    a->offset = offset;
    a->data = base_data + offset;
    a->owns = false;
    return reinterpret_cast<PyObject *>(a);
}

// A new array of the pool; nullptr without an exception when the pool refuses (ops.py asks again and reports why).
PyObject *new_array(PyObject *dev, PyObject *shape /*stolen, may be null*/, int dtype, int64_t bytes) {
    if (!shape) return nullptr;
    void *p = nullptr;
    nvc_device *h = reinterpret_cast<DeviceObject *>(dev)->handle;
    if (!h || L.nvc_alloc(h, bytes > 0 ? (size_t)bytes : 1, &p) != NVC_OK) {
        Py_DECREF(shape);
        return nullptr;
    }
    ArrayObject *a = reinterpret_cast<ArrayObject *>(array_class->tp_alloc(array_class, 0));
    if (!a) {
        Py_DECREF(shape);
        L.nvc_free(h, p);
        return nullptr;
    }
    a->dev = Py_NewRef(dev);
    a->shape = shape;
    a->base = nullptr;
    a->dtype = dtype;
    a->offset = 0;
    a->data = static_cast<char *>(p);
    a->owns = true;
    return reinterpret_cast<PyObject *>(a);
}
PyObject *shape1(int64_t a) { return Py_BuildValue("(L)", (long long)a); }
// The first `lead` dimensions of a, then the given ones (up to two; -1: none).
PyObject *shape_with(const ArrayObject *a, Py_ssize_t lead, int64_t d0, int64_t d1 = -1) {
    const Py_ssize_t extra = (d0 >= 0) + (d1 >= 0);
    PyObject *t = PyTuple_New(lead + extra);
    if (!t) return nullptr;
    for (Py_ssize_t i = 0; i < lead; i++) PyTuple_SET_ITEM(t, i, Py_NewRef(PyTuple_GET_ITEM(a->shape, i)));
    if (d0 >= 0) PyTuple_SET_ITEM(t, lead, PyLong_FromLongLong(d0));
    if (d1 >= 0) PyTuple_SET_ITEM(t, lead + 1, PyLong_FromLongLong(d1));
    return t;
}

// Array(dev, shape, dtype, _base=None, _offset=0)
int array_init(PyObject *self, PyObject *args, PyObject *kw) {
    static const char *names[] = {"dev", "shape", "dtype", "_base", "_offset", nullptr};
    PyObject *dev, *shape, *base = Py_None;
    int dtype;
    Py_ssize_t offset = 0;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "OOi|On", const_cast<char **>(names), &dev, &shape, &dtype, &base, &offset)) return -1;
    if (!PyObject_TypeCheck(dev, &DeviceType)) {
        PyErr_SetString(PyExc_TypeError, "an array needs a Device");
        return -1;
    }
    ArrayObject *a = arr(self);
    if (a->dev) {
        PyErr_SetString(PyExc_TypeError, "an array is initialized once");
        return -1;
    }
    if (item_size(dtype) == 0) {
        PyErr_Format(PyExc_KeyError, "%d is no dtype code", dtype);
        return -1;
    }
    a->shape = PySequence_Tuple(shape);
    if (!a->shape) return -1;
    int64_t bytes = item_size(dtype);
    for (Py_ssize_t i = 0; i < rank(a); i++) {
        const int64_t d = dim(a, i);
        if (d == -1 && PyErr_Occurred()) return -1;
        if (d < 0) {
            PyErr_Format(PyExc_ValueError, "an array of shape %R", a->shape);
            return -1;
        }
        if (__builtin_mul_overflow(bytes, d, &bytes)) {
            PyErr_Format(PyExc_OverflowError, "an array of shape %R", a->shape);
            return -1;
        }
    }
    a->dtype = dtype;
    a->dev = Py_NewRef(dev);
    a->offset = offset;
    if (base == Py_None) return 1;  // (the caller allocates: see array_init_py)
    a->base = Py_NewRef(base);
    if (is_array(base)) {
        a->data = arr(base)->data + offset;
        return 0;
    }
    Ref ptr(PyObject_GetAttr(base, s_ptr));
    Ref value(ptr ? PyObject_GetAttr(ptr.o, s_value) : nullptr);
    if (!value) return -1;
    a->data = static_cast<char *>(PyLong_AsVoidPtr(value.o)) + offset;
    return PyErr_Occurred() ? -1 : 0;
}
int array_init_py(PyObject *self, PyObject *args, PyObject *kw) {
    const int rc = array_init(self, args, kw);
    if (rc != 1) return rc;
    ArrayObject *a = arr(self);
    const int64_t bytes = size_of(a) * item_size(a->dtype);
    if (PyErr_Occurred()) return -1;
    void *p = nullptr;
    nvc_device *h = handle_of(a);
    const int32_t status = h ? L.nvc_alloc(h, bytes > 0 ? (size_t)bytes : 1, &p) : (int32_t)NVC_ERR_INVALID_ARGUMENT;
    if (status != NVC_OK) {  // the caller turns the status into its own exception
        PyErr_Format(PyExc_MemoryError, "nvc:%d", (int)status);
        return -1;
    }
    a->data = static_cast<char *>(p);
    a->owns = true;
    return 0;
}
void array_dealloc(PyObject *self) {
    ArrayObject *a = arr(self);
    PyTypeObject *type = Py_TYPE(self);
    if (a->owns && a->dev) {
        nvc_device *h = handle_of(a);
        if (h) L.nvc_free(h, a->data);
    }
    Py_CLEAR(a->base);
    Py_CLEAR(a->dev);
    Py_CLEAR(a->shape);
    type->tp_free(self);
}
PyObject *array_address(PyObject *self, void *) { return PyLong_FromVoidPtr(arr(self)->data); }
PyObject *array_ptr_or_none(PyObject *self, void *) {
    if (arr(self)->base) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(arr(self)->data);
}
PyObject *array_base(PyObject *self, void *) { return Py_NewRef(arr(self)->base ? arr(self)->base : Py_None); }
PyObject *array_size(PyObject *self, void *) { return PyLong_FromLongLong(size_of(arr(self))); }
PyObject *array_ndim(PyObject *self, void *) { return PyLong_FromSsize_t(rank(arr(self))); }
PyObject *array_nbytes(PyObject *self, void *) { return PyLong_FromLongLong(size_of(arr(self)) * item_size(arr(self)->dtype)); }
PyObject *array_itemsize(PyObject *self, void *) { return PyLong_FromLong(item_size(arr(self)->dtype)); }

PyObject *root_of(ArrayObject *a) { return a->base ? a->base : reinterpret_cast<PyObject *>(a); }
PyObject *view(ArrayObject *a, PyObject *shape /*stolen*/, int64_t more) {
    return view_of(Py_TYPE(reinterpret_cast<PyObject *>(a)), a->dev, shape, a->dtype, root_of(a), a->offset + more, a->data - a->offset);
}

// reshape(*dims) or reshape(dims); one dimension may be -1
PyObject *array_reshape(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    ArrayObject *a = arr(self);
    Ref given(n == 1 && (PyTuple_Check(args[0]) || PyList_Check(args[0])) ? PySequence_Tuple(args[0]) : nullptr);
    if (!given) {
        if (PyErr_Occurred()) return nullptr;
        given.o = PyTuple_New(n);
        if (!given) return nullptr;
        for (Py_ssize_t i = 0; i < n; i++) PyTuple_SET_ITEM(given.o, i, Py_NewRef(args[i]));
    }
    const Py_ssize_t dims = PyTuple_GET_SIZE(given.o);
    int64_t known = 1;
    Py_ssize_t open_at = -1;
    for (Py_ssize_t i = 0; i < dims; i++) {
        const int64_t d = PyLong_AsLongLong(PyTuple_GET_ITEM(given.o, i));
        if (d == -1 && PyErr_Occurred()) return nullptr;
        if (d == -1) open_at = i;
        else known *= d;
    }
    const int64_t size = size_of(a);
    Ref shape(PyTuple_New(dims));
    if (!shape) return nullptr;
    int64_t total = 1;
    for (Py_ssize_t i = 0; i < dims; i++) {
        int64_t d = PyLong_AsLongLong(PyTuple_GET_ITEM(given.o, i));
        if (d == -1) d = i == open_at && known ? size / known : 0;
        total *= d;
        PyTuple_SET_ITEM(shape.o, i, PyLong_FromLongLong(d));
    }
    if (total != size) {
        PyErr_Format(PyExc_AssertionError, "(%R, %R)", shape.o, a->shape);
        return nullptr;
    }
    return view(a, shape.release(), 0);
}

// a[i], a[lo:hi]: a view along the leading axis
PyObject *array_getitem(PyObject *self, PyObject *index) {
    ArrayObject *a = arr(self);
    const Py_ssize_t r = rank(a);
    if (r < 1) {
        PyErr_SetString(PyExc_IndexError, "an array without dimensions has no items");
        return nullptr;
    }
    int64_t inner = 1;
    for (Py_ssize_t i = 1; i < r; i++) inner *= dim(a, i);
    const int64_t n = dim(a, 0), step_bytes = inner * item_size(a->dtype);
    if (PySlice_Check(index)) {
        Py_ssize_t start, stop, step;
        if (PySlice_Unpack(index, &start, &stop, &step) < 0) return nullptr;
        const Py_ssize_t len = PySlice_AdjustIndices((Py_ssize_t)n, &start, &stop, step);
        if (step != 1) {
            PyErr_SetNone(PyExc_AssertionError);
            return nullptr;
        }
        Ref shape(PyTuple_New(r));
        if (!shape) return nullptr;
        PyTuple_SET_ITEM(shape.o, 0, PyLong_FromSsize_t(len));
        for (Py_ssize_t i = 1; i < r; i++) PyTuple_SET_ITEM(shape.o, i, Py_NewRef(PyTuple_GET_ITEM(a->shape, i)));
        return view(a, shape.release(), start * step_bytes);
    }
    Ref as_int(PyNumber_Long(index));
    if (!as_int) return nullptr;
    int64_t i = PyLong_AsLongLong(as_int.o);
    if (i == -1 && PyErr_Occurred()) return nullptr;
    if (n == 0) {
        PyErr_SetString(PyExc_ZeroDivisionError, "integer modulo by zero");
        return nullptr;
    }
    i %= n;
    if (i < 0) i += n;
    PyObject *shape = PyTuple_GetSlice(a->shape, 1, r);
    return shape ? view(a, shape, i * step_bytes) : nullptr;
}

PyMethodDef array_methods[] = {
    {"reshape", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(array_reshape)), METH_FASTCALL, "The same values in another shape."},
    {"__getitem__", array_getitem, METH_O | METH_COEXIST, "Leading-axis integer or slice (a contiguous view)."},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef array_members[] = {{"dev", T_OBJECT_EX, offsetof(ArrayObject, dev), READONLY, nullptr},
                               {"shape", T_OBJECT_EX, offsetof(ArrayObject, shape), READONLY, nullptr},
                               {"dtype", T_INT, offsetof(ArrayObject, dtype), READONLY, nullptr},
                               {"_offset", T_PYSSIZET, offsetof(ArrayObject, offset), READONLY, nullptr},
                               {nullptr, 0, 0, 0, nullptr}};
PyGetSetDef array_getset[] = {{"_address", array_address, nullptr, nullptr, nullptr}, {"_ptr", array_ptr_or_none, nullptr, nullptr, nullptr},
                              {"_base", array_base, nullptr, nullptr, nullptr},       {"size", array_size, nullptr, nullptr, nullptr},
                              {"ndim", array_ndim, nullptr, nullptr, nullptr},        {"nbytes", array_nbytes, nullptr, nullptr, nullptr},
                              {"itemsize", array_itemsize, nullptr, nullptr, nullptr}, {nullptr, nullptr, nullptr, nullptr, nullptr}};

PyObject *device_set_handle(PyObject *self, PyObject *value) {
    void *h = value == Py_None ? nullptr : PyLong_AsVoidPtr(value);
    if (PyErr_Occurred()) return nullptr;
    reinterpret_cast<DeviceObject *>(self)->handle = static_cast<nvc_device *>(h);
    Py_RETURN_NONE;
}
PyMethodDef device_methods[] = {{"_set_handle", device_set_handle, METH_O, "The library's handle as an integer; None once it is closed."},
                                {nullptr, nullptr, 0, nullptr}};

// ── quantized operands ──────────────────────────────────────────────────────────────────
// A Quantized's parts (references held) in the forms the fast paths take.
struct Packed {
    Ref weight, scales, biases, quant_obj, global;
    nvc_quant quant{};
    bool ok = false;
    ArrayObject *w() const { return weight.array(); }
    ArrayObject *s() const { return scales.array(); }
    ArrayObject *b() const { return biases.o == Py_None ? nullptr : biases.array(); }
    ArrayObject *g() const { return global.o == Py_None ? nullptr : global.array(); }
};
bool read_quant(PyObject *o, nvc_quant &q) {
    Ref mode(PyObject_GetAttr(o, s_mode)), group(PyObject_GetAttr(o, s_group)), bits(PyObject_GetAttr(o, s_bits));
    if (!mode || !group || !bits || !PyLong_Check(group.o) || !PyLong_Check(bits.o)) return false;
    q.mode = -1;
    for (int i = 0; i < 4; i++)
        if (mode.o == modes[i]) q.mode = i;
    q.group_size = (int32_t)PyLong_AsLong(group.o);
    q.bits = (int32_t)PyLong_AsLong(bits.o);
    return q.mode >= 0 && q.group_size > 0 && q.bits > 0 && !PyErr_Occurred();
}
// Codes uint32 [..., rows, words] with scales (and, affine, biases) [..., rows, cols / group] of one float type.
bool read_packed(PyObject *o, Packed &p) {
    if (reinterpret_cast<PyObject *>(Py_TYPE(o)) != quantized_class) return false;
    p.weight.o = PyObject_GetAttr(o, s_weight);
    p.scales.o = PyObject_GetAttr(o, s_scales);
    p.biases.o = PyObject_GetAttr(o, s_biases);
    p.quant_obj.o = PyObject_GetAttr(o, s_quant);
    p.global.o = PyObject_GetAttr(o, s_global);
    if (!p.weight || !p.scales || !p.biases || !p.quant_obj || !p.global) return false;
    if (!is_array(p.weight.o) || !is_array(p.scales.o) || (p.biases.o != Py_None && !is_array(p.biases.o)) ||
        (p.global.o != Py_None && !is_array(p.global.o)) || !read_quant(p.quant_obj.o, p.quant))
        return false;
    const ArrayObject *w = p.w(), *s = p.s();
    const Py_ssize_t r = rank(w);
    if (w->dtype != NVC_U32 || r < 2 || rank(s) != r) return false;
    for (Py_ssize_t i = 0; i + 1 < r; i++)
        if (dim(w, i) != dim(s, i)) return false;
    const int64_t cols = dim(w, -1) * 32 / p.quant.bits;
    if (cols % p.quant.group_size != 0 || dim(s, -1) != cols / p.quant.group_size) return false;
    if (p.quant.mode == NVC_AFFINE) {
        if (!p.b() || !is_float(s->dtype) || p.b()->dtype != s->dtype || !same_shape(s, p.b())) return false;
    } else if (p.b() || s->dtype != NVC_U8) {
        return false;
    }
    return s->dev == w->dev && (!p.b() || p.b()->dev == w->dev) && (!p.g() || p.g()->dev == w->dev);
}
int64_t cols_of(const Packed &p) { return dim(p.w(), -1) * 32 / p.quant.bits; }
const void *data_of(const ArrayObject *a) { return a ? a->data : nullptr; }

template <class F> int32_t unlocked(F f) {  // a launch may wait for room in the queue: other threads go on meanwhile
    int32_t rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}
#define DECLINE_UNLESS(cond) \
    do {                     \
        if (!(cond)) return decline(); \
    } while (0)
#define FINISH(result, call)                    \
    do {                                        \
        if (unlocked([&] { return (call); }) != NVC_OK) return decline(); \
        return (result).release();              \
    } while (0)

// ── operators ───────────────────────────────────────────────────────────────────────────
// quantized_matmul(x, q, transpose)
PyObject *f_quantized_matmul(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed p;
    DECLINE_UNLESS(n == 3 && is_array(a[0]) && read_packed(a[1], p));
    const ArrayObject *x = arr(a[0]), *w = p.w(), *g = p.g();
    const int transpose = PyObject_IsTrue(a[2]);
    const Py_ssize_t xr = rank(x);
    DECLINE_UNLESS(transpose >= 0 && rank(w) == 2 && xr >= 1 && is_float(x->dtype) && x->dev == w->dev);
    DECLINE_UNLESS(p.quant.mode != NVC_AFFINE || p.s()->dtype == x->dtype);
    DECLINE_UNLESS(!g || (p.quant.mode == NVC_NVFP4 && transpose && xr <= 2 && g->dtype == NVC_F32 && size_of(g) == 1));
    const int64_t rows = dim(w, 0), cols = cols_of(p), K = transpose ? cols : rows, N = transpose ? rows : cols;
    DECLINE_UNLESS(dim(x, -1) == K);
    const int64_t M = xr == 1 ? 1 : dim(x, -2);
    int64_t batch = 1;
    for (Py_ssize_t i = 0; i + 2 < xr; i++) batch *= dim(x, i);
    nvc_device *h = handle_of(x);
    Ref y(new_array(x->dev, shape_with(x, xr - 1, N), x->dtype, batch * M * N * item_size(x->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_quantized_matmul(h, &p.quant, x->dtype, transpose, x->data, reinterpret_cast<const uint32_t *>(w->data), p.s()->data, data_of(p.b()),
                                     static_cast<const float *>(data_of(g)), M, N, K, K, batch, M * K, 0, 0, y.array()->data));
}

// gather_qmm(x, q, lhs, rhs, transpose, sorted, offsets)
PyObject *f_gather_qmm(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed p;
    DECLINE_UNLESS(n == 7 && is_array(a[0]) && is_array(a[3]) && (a[2] == Py_None || is_array(a[2])) && (a[6] == Py_None || is_array(a[6])) &&
                   read_packed(a[1], p));
    const ArrayObject *x = arr(a[0]), *w = p.w(), *g = p.g(), *rhs = arr(a[3]), *lhs = a[2] == Py_None ? nullptr : arr(a[2]),
                      *offs = a[6] == Py_None ? nullptr : arr(a[6]);
    const int transpose = PyObject_IsTrue(a[4]), sorted = PyObject_IsTrue(a[5]);
    const Py_ssize_t xr = rank(x), rr = rank(rhs);
    DECLINE_UNLESS(transpose >= 0 && sorted >= 0 && xr >= 2 && is_float(x->dtype) && x->dev == w->dev && rhs->dev == w->dev);
    DECLINE_UNLESS((rhs->dtype == NVC_U32 || rhs->dtype == NVC_I32) && (!lhs || ((lhs->dtype == NVC_U32 || lhs->dtype == NVC_I32) && lhs->dev == w->dev)));
    DECLINE_UNLESS(p.quant.mode != NVC_AFFINE || p.s()->dtype == x->dtype);
    int64_t experts = 1, x_batches = 1, count = 1;
    for (Py_ssize_t i = 0; i + 2 < rank(w); i++) experts *= dim(w, i);
    for (Py_ssize_t i = 0; i + 2 < xr; i++) x_batches *= dim(x, i);
    for (Py_ssize_t i = 0; i < rr; i++) count *= dim(rhs, i);
    if (g) {
        DECLINE_UNLESS(p.quant.mode == NVC_NVFP4 && g->dtype == NVC_F32 && rank(g) == rank(w) - 2);
        for (Py_ssize_t i = 0; i < rank(g); i++) DECLINE_UNLESS(dim(g, i) == dim(w, i));
    }
    if (lhs) {
        DECLINE_UNLESS(same_shape(lhs, rhs));
    } else {  // the activations' batches in order: the index shape is theirs
        DECLINE_UNLESS(rr == xr - 2);
        for (Py_ssize_t i = 0; i < rr; i++) DECLINE_UNLESS(dim(rhs, i) == dim(x, i));
    }
    const int64_t rows = dim(w, -2), cols = cols_of(p), K = transpose ? cols : rows, N = transpose ? rows : cols, M = dim(x, -2);
    DECLINE_UNLESS(dim(x, -1) == K);
    nvc_device *h = handle_of(x);
    Ref y(new_array(x->dev, shape_with(rhs, rr, M, N), x->dtype, count * M * N * item_size(x->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_gather_qmm(h, &p.quant, x->dtype, transpose, x->data, reinterpret_cast<const uint32_t *>(w->data), p.s()->data, data_of(p.b()),
                               static_cast<const float *>(data_of(g)), static_cast<const uint32_t *>(data_of(lhs)),
                               reinterpret_cast<const uint32_t *>(rhs->data), static_cast<const int32_t *>(data_of(offs)), sorted, count, x_batches, M, N,
                               K, experts, y.array()->data));
}

// qqmm(x, q, prepared)
PyObject *f_qqmm(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed p;
    DECLINE_UNLESS(n == 3 && is_array(a[0]) && (a[2] == Py_None || is_array(a[2])) && read_packed(a[1], p));
    const ArrayObject *x = arr(a[0]), *w = p.w(), *prepared = a[2] == Py_None ? nullptr : arr(a[2]);
    DECLINE_UNLESS((p.quant.mode == NVC_NVFP4 || p.quant.mode == NVC_MXFP4) && !p.g() && x->dtype == NVC_BF16 && rank(x) >= 1 && rank(w) == 2 && x->dev == w->dev);
    const int64_t K = dim(x, -1), N = dim(w, 0);
    DECLINE_UNLESS(dim(w, 1) * 8 == K && K > 0);
    const int64_t M = size_of(x) / K;
    nvc_device *h = handle_of(x);
    Ref y(new_array(x->dev, shape_with(x, rank(x) - 1, N), NVC_BF16, M * N * 2));
    DECLINE_UNLESS(h && y);
    const uint32_t *codes = reinterpret_cast<const uint32_t *>(w->data);
    FINISH(y, prepared ? L.nvc_qqmm_prepared(h, &p.quant, NVC_BF16, x->data, codes, prepared->data, M, N, K, y.array()->data)
                       : L.nvc_qqmm(h, &p.quant, NVC_BF16, x->data, codes, p.s()->data, M, N, K, y.array()->data));
}

// quantize(w, quant): (codes, scales, biases or None)
PyObject *f_quantize(PyObject *, PyObject *const *a, Py_ssize_t n) {
    nvc_quant q;
    DECLINE_UNLESS(n == 2 && is_array(a[0]) && read_quant(a[1], q));
    const ArrayObject *w = arr(a[0]);
    const Py_ssize_t r = rank(w);
    DECLINE_UNLESS(is_float(w->dtype) && r >= 2);
    const int64_t cols = dim(w, -1), size = size_of(w);
    DECLINE_UNLESS(cols > 0 && cols % q.group_size == 0);
    const bool affine = q.mode == NVC_AFFINE;
    const int64_t groups = size / q.group_size;
    nvc_device *h = handle_of(w);
    Ref codes(new_array(w->dev, shape_with(w, r - 1, cols * q.bits / 32), NVC_U32, size / cols * (cols * q.bits / 32) * 4));
    Ref scales(new_array(w->dev, shape_with(w, r - 1, cols / q.group_size), affine ? w->dtype : (int)NVC_U8, groups * (affine ? item_size(w->dtype) : 1)));
    Ref biases(affine ? new_array(w->dev, shape_with(w, r - 1, cols / q.group_size), w->dtype, groups * item_size(w->dtype)) : Py_NewRef(Py_None));
    DECLINE_UNLESS(h && codes && scales && biases);
    Ref out(PyTuple_Pack(3, codes.o, scales.o, biases.o));
    if (!out) return nullptr;
    FINISH(out, L.nvc_quantize(h, &q, w->dtype, w->data, size / cols, cols, nullptr, reinterpret_cast<uint32_t *>(codes.array()->data), scales.array()->data,
                               affine ? biases.array()->data : nullptr));
}

// dequantize(q) into the scales' type (bfloat16 for the floating-point modes)
PyObject *f_dequantize(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed p;
    DECLINE_UNLESS(n == 1 && read_packed(a[0], p) && !p.g());
    const ArrayObject *w = p.w();
    const int dtype = p.quant.mode == NVC_AFFINE ? p.s()->dtype : (int)NVC_BF16;
    const int64_t cols = cols_of(p), words = dim(w, -1);
    DECLINE_UNLESS(words > 0);
    const int64_t rows = size_of(w) / words;
    nvc_device *h = handle_of(w);
    Ref y(new_array(w->dev, shape_with(w, rank(w) - 1, cols), dtype, rows * cols * item_size(dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_dequantize(h, &p.quant, dtype, reinterpret_cast<const uint32_t *>(w->data), p.s()->data, data_of(p.b()), nullptr, rows, cols,
                               y.array()->data, 0));
}

// quantized_embedding(q, ids)
PyObject *f_quantized_embedding(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed p;
    DECLINE_UNLESS(n == 2 && is_array(a[1]) && read_packed(a[0], p) && !p.g());
    const ArrayObject *w = p.w(), *ids = arr(a[1]);
    DECLINE_UNLESS(rank(w) == 2 && ids->dtype == NVC_U32 && ids->dev == w->dev);
    const int dtype = p.quant.mode == NVC_AFFINE ? p.s()->dtype : (int)NVC_BF16;
    const int64_t cols = cols_of(p), count = size_of(ids);
    nvc_device *h = handle_of(w);
    Ref y(new_array(w->dev, shape_with(ids, rank(ids), cols), dtype, count * cols * item_size(dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_quantized_embedding(h, &p.quant, dtype, reinterpret_cast<const uint32_t *>(w->data), p.s()->data, data_of(p.b()), dim(w, 0), cols,
                                        reinterpret_cast<const uint32_t *>(ids->data), count, y.array()->data));
}

// sorted_offsets(indices, groups)
PyObject *f_sorted_offsets(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 2 && is_array(a[0]) && PyLong_Check(a[1]));
    const ArrayObject *idx = arr(a[0]);
    const int64_t groups = PyLong_AsLongLong(a[1]);
    DECLINE_UNLESS(idx->dtype == NVC_U32 && groups >= 0);
    nvc_device *h = handle_of(idx);
    Ref y(new_array(idx->dev, shape1(groups), NVC_I32, groups * 4));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_sorted_offsets(h, reinterpret_cast<const uint32_t *>(idx->data), size_of(idx), groups, reinterpret_cast<int32_t *>(y.array()->data)));
}

// moe_route(probs, k, normalize): (indices, scores)
PyObject *f_moe_route(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 3 && is_array(a[0]) && PyLong_Check(a[1]));
    const ArrayObject *probs = arr(a[0]);
    const int64_t k = PyLong_AsLongLong(a[1]);
    const int normalize = PyObject_IsTrue(a[2]);
    DECLINE_UNLESS(is_float(probs->dtype) && rank(probs) >= 1 && normalize >= 0 && k >= 1 && k <= dim(probs, -1));
    const int64_t experts = dim(probs, -1), rows = size_of(probs) / experts;
    const Py_ssize_t lead = rank(probs) - 1;
    nvc_device *h = handle_of(probs);
    Ref idx(new_array(probs->dev, shape_with(probs, lead, k), NVC_U32, rows * k * 4));
    Ref scores(new_array(probs->dev, shape_with(probs, lead, k), probs->dtype, rows * k * item_size(probs->dtype)));
    DECLINE_UNLESS(h && idx && scores);
    Ref out(PyTuple_Pack(2, idx.o, scores.o));
    if (!out) return nullptr;
    FINISH(out, L.nvc_moe_route(h, probs->dtype, probs->data, rows, experts, k, normalize, reinterpret_cast<uint32_t *>(idx.array()->data), scores.array()->data));
}

// weighted_sum(x, w)
PyObject *f_weighted_sum(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 2 && is_array(a[0]) && is_array(a[1]));
    const ArrayObject *x = arr(a[0]), *w = arr(a[1]);
    const Py_ssize_t r = rank(x);
    DECLINE_UNLESS(r >= 2 && rank(w) == r - 1 && is_float(x->dtype) && w->dtype == x->dtype && w->dev == x->dev);
    for (Py_ssize_t i = 0; i + 1 < r; i++) DECLINE_UNLESS(dim(x, i) == dim(w, i));
    const int64_t k = dim(x, -2), d = dim(x, -1);
    DECLINE_UNLESS(k > 0 && d > 0);
    const int64_t rows = size_of(w) / k;
    nvc_device *h = handle_of(x);
    Ref y(new_array(x->dev, shape_with(x, r - 2, d), x->dtype, rows * d * item_size(x->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_weighted_sum(h, x->dtype, x->data, w->data, rows, k, d, y.array()->data));
}

// expert_bias_add(y, bias, indices): y itself
PyObject *f_expert_bias_add(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 3 && is_array(a[0]) && is_array(a[1]) && is_array(a[2]));
    const ArrayObject *y = arr(a[0]), *bias = arr(a[1]), *idx = arr(a[2]);
    DECLINE_UNLESS(rank(bias) == 2 && rank(y) >= 2 && is_float(y->dtype) && bias->dtype == y->dtype && idx->dtype == NVC_U32 && bias->dev == y->dev &&
                   idx->dev == y->dev);
    const int64_t width = dim(y, -1);
    DECLINE_UNLESS(width > 0 && dim(bias, 1) == width);
    const int64_t rows = size_of(y) / width;
    DECLINE_UNLESS(size_of(idx) == rows);
    nvc_device *h = handle_of(y);
    DECLINE_UNLESS(h);
    Ref same(Py_NewRef(a[0]));
    FINISH(same, L.nvc_expert_bias_add(h, y->dtype, y->data, bias->data, reinterpret_cast<const uint32_t *>(idx->data), rows, width, dim(bias, 0)));
}

// moe_sort(indices, experts): (order, restore, tokens, sorted, offsets)
PyObject *f_moe_sort(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 2 && is_array(a[0]) && PyLong_Check(a[1]));
    const ArrayObject *idx = arr(a[0]);
    const int64_t experts = PyLong_AsLongLong(a[1]);
    DECLINE_UNLESS(idx->dtype == NVC_U32 && rank(idx) >= 1 && dim(idx, -1) >= 1 && experts >= 0);
    const int64_t pairs = size_of(idx);
    nvc_device *h = handle_of(idx);
    Ref order(new_array(idx->dev, shape1(pairs), NVC_U32, pairs * 4)), restore(new_array(idx->dev, shape1(pairs), NVC_U32, pairs * 4));
    Ref tokens(new_array(idx->dev, shape1(pairs), NVC_U32, pairs * 4)), sorted(new_array(idx->dev, shape1(pairs), NVC_U32, pairs * 4));
    Ref offs(new_array(idx->dev, shape1(experts), NVC_I32, experts * 4));
    DECLINE_UNLESS(h && order && restore && tokens && sorted && offs);
    Ref out(PyTuple_Pack(5, order.o, restore.o, tokens.o, sorted.o, offs.o));
    if (!out) return nullptr;
    auto u32 = [](const Ref &r) { return reinterpret_cast<uint32_t *>(r.array()->data); };
    FINISH(out, L.nvc_moe_sort(h, reinterpret_cast<const uint32_t *>(idx->data), pairs, dim(idx, -1), experts, u32(order), u32(restore), u32(tokens),
                               u32(sorted), reinterpret_cast<int32_t *>(offs.array()->data)));
}

// take_rows(src, indices)
PyObject *f_take_rows(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 2 && is_array(a[0]) && is_array(a[1]));
    const ArrayObject *src = arr(a[0]), *idx = arr(a[1]);
    DECLINE_UNLESS(rank(src) >= 1 && dim(src, 0) > 0 && idx->dtype == NVC_U32 && idx->dev == src->dev);
    const int64_t rows = dim(src, 0), row_bytes = size_of(src) / rows * item_size(src->dtype), count = size_of(idx);
    Ref shape(PyTuple_New(rank(src)));
    if (!shape) return nullptr;
    PyTuple_SET_ITEM(shape.o, 0, PyLong_FromLongLong(count));
    for (Py_ssize_t i = 1; i < rank(src); i++) PyTuple_SET_ITEM(shape.o, i, Py_NewRef(PyTuple_GET_ITEM(src->shape, i)));
    nvc_device *h = handle_of(src);
    Ref y(new_array(src->dev, shape.release(), src->dtype, count * row_bytes));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_take_rows(h, src->data, rows, row_bytes, reinterpret_cast<const uint32_t *>(idx->data), count, y.array()->data));
}

bool norm_args(const ArrayObject *x, PyObject *weight) {
    if (rank(x) < 1 || !is_float(x->dtype) || dim(x, -1) < 1) return false;
    if (weight == Py_None) return true;
    return is_array(weight) && arr(weight)->dtype == x->dtype && rank(arr(weight)) == 1 && dim(arr(weight), 0) == dim(x, -1) && arr(weight)->dev == x->dev;
}
// rms_norm(x, weight, eps)
PyObject *f_rms_norm(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 3 && is_array(a[0]) && norm_args(arr(a[0]), a[1]));
    const ArrayObject *x = arr(a[0]);
    const double eps = PyFloat_AsDouble(a[2]);
    DECLINE_UNLESS(!PyErr_Occurred());
    const int64_t d = dim(x, -1), size = size_of(x);
    nvc_device *h = handle_of(x);
    Ref y(new_array(x->dev, Py_NewRef(x->shape), x->dtype, size * item_size(x->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_rms_norm(h, x->dtype, x->data, a[1] == Py_None ? nullptr : arr(a[1])->data, (float)eps, size / d, d, y.array()->data));
}
// add_rms_norm(x, residual, weight, eps): (sum, normalized)
PyObject *f_add_rms_norm(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS(n == 4 && is_array(a[0]) && is_array(a[1]) && norm_args(arr(a[0]), a[2]));
    const ArrayObject *x = arr(a[0]), *r = arr(a[1]);
    const double eps = PyFloat_AsDouble(a[3]);
    DECLINE_UNLESS(!PyErr_Occurred() && r->dtype == x->dtype && r->dev == x->dev && same_shape(x, r));
    const int64_t d = dim(x, -1), size = size_of(x);
    nvc_device *h = handle_of(x);
    Ref sum(new_array(x->dev, Py_NewRef(x->shape), x->dtype, size * item_size(x->dtype))), y(new_array(x->dev, Py_NewRef(x->shape), x->dtype, size * item_size(x->dtype)));
    DECLINE_UNLESS(h && sum && y);
    Ref out(PyTuple_Pack(2, sum.o, y.o));
    if (!out) return nullptr;
    FINISH(out, L.nvc_add_rms_norm(h, x->dtype, x->data, r->data, a[2] == Py_None ? nullptr : arr(a[2])->data, (float)eps, size / d, d, sum.array()->data,
                                   y.array()->data));
}

// swiglu(gate, up) and swiglu(gate, up, alpha, limit)
PyObject *f_swiglu(PyObject *, PyObject *const *a, Py_ssize_t n) {
    DECLINE_UNLESS((n == 2 || n == 4) && is_array(a[0]) && is_array(a[1]));
    const ArrayObject *g = arr(a[0]), *u = arr(a[1]);
    DECLINE_UNLESS(is_float(g->dtype) && u->dtype == g->dtype && u->dev == g->dev && same_shape(g, u));
    double alpha = 0, limit = 0;
    if (n == 4) {
        alpha = PyFloat_AsDouble(a[2]);
        limit = PyFloat_AsDouble(a[3]);
        DECLINE_UNLESS(!PyErr_Occurred());
    }
    const int64_t size = size_of(g);
    nvc_device *h = handle_of(g);
    Ref y(new_array(g->dev, Py_NewRef(g->shape), g->dtype, size * item_size(g->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, n == 2 ? L.nvc_swiglu(h, g->dtype, g->data, u->data, size, y.array()->data)
                     : L.nvc_swiglu_oai(h, g->dtype, g->data, u->data, (float)alpha, (float)limit, size, y.array()->data));
}

// quantized_attention(q, k, v, scale, sinks, length, causal)
PyObject *f_quantized_attention(PyObject *, PyObject *const *a, Py_ssize_t n) {
    Packed k, v;
    DECLINE_UNLESS(n == 7 && is_array(a[0]) && (a[4] == Py_None || is_array(a[4])) && read_packed(a[1], k) && read_packed(a[2], v));
    const ArrayObject *q = arr(a[0]), *sinks = a[4] == Py_None ? nullptr : arr(a[4]);
    DECLINE_UNLESS(k.quant.mode == NVC_AFFINE && v.quant.mode == NVC_AFFINE && k.quant.group_size == v.quant.group_size && k.quant.bits == v.quant.bits);
    DECLINE_UNLESS(rank(q) == 4 && rank(k.w()) == 4 && same_shape(k.w(), v.w()) && k.s()->dtype == q->dtype && v.s()->dtype == q->dtype &&
                   k.w()->dev == q->dev && v.w()->dev == q->dev);
    const double scale = PyFloat_AsDouble(a[3]);
    const int causal = PyObject_IsTrue(a[6]);
    const int64_t B = dim(q, 0), Hq = dim(q, 1), rows = dim(q, 2), D = dim(q, 3), Hkv = dim(k.w(), 1), cap = dim(k.w(), 2);
    const int64_t S = a[5] == Py_None ? cap : PyLong_AsLongLong(a[5]);
    DECLINE_UNLESS(!PyErr_Occurred() && causal >= 0 && dim(k.w(), 0) == B && cols_of(k) == D && S >= 0 && S <= cap);
    DECLINE_UNLESS(!sinks || (rank(sinks) == 1 && dim(sinks, 0) == Hq && sinks->dtype == q->dtype && sinks->dev == q->dev));
    nvc_device *h = handle_of(q);
    Ref y(new_array(q->dev, Py_NewRef(q->shape), q->dtype, size_of(q) * item_size(q->dtype)));
    DECLINE_UNLESS(h && y);
    FINISH(y, L.nvc_quantized_attention(h, &k.quant, q->dtype, q->data, reinterpret_cast<const uint32_t *>(k.w()->data), k.s()->data, k.b()->data,
                                        reinterpret_cast<const uint32_t *>(v.w()->data), v.s()->data, v.b()->data, data_of(sinks), B, Hq, Hkv, rows, S, D,
                                        cap, (float)scale, causal, y.array()->data));
}

// bind({name: address}): the library's functions
PyObject *f_bind(PyObject *, PyObject *table) {
    if (!PyDict_Check(table)) {
        PyErr_SetString(PyExc_TypeError, "bind: a dict of addresses");
        return nullptr;
    }
#define NVC_BIND(name)                                                              \
    {                                                                               \
        PyObject *v = PyDict_GetItemString(table, #name);                           \
        if (!v) {                                                                   \
            PyErr_SetString(PyExc_KeyError, #name);                                 \
            return nullptr;                                                         \
        }                                                                           \
        L.name = reinterpret_cast<decltype(L.name)>(PyLong_AsVoidPtr(v));           \
        if (PyErr_Occurred()) return nullptr;                                       \
    }
    NVC_BOUND(NVC_BIND)
#undef NVC_BIND
    Py_RETURN_NONE;
}
// register(Array, Quantized, (affine, mxfp4, mxfp8, nvfp4)): the classes of ops.py
PyObject *f_register(PyObject *, PyObject *args) {
    PyObject *array, *quantized, *m[4];
    if (!PyArg_ParseTuple(args, "OO(OOOO)", &array, &quantized, &m[0], &m[1], &m[2], &m[3])) return nullptr;
    if (!PyType_Check(array) || !PyType_IsSubtype(reinterpret_cast<PyTypeObject *>(array), &ArrayType)) {
        PyErr_SetString(PyExc_TypeError, "register: a subclass of ArrayBase");
        return nullptr;
    }
    array_class = reinterpret_cast<PyTypeObject *>(Py_NewRef(array));
    quantized_class = Py_NewRef(quantized);
    for (int i = 0; i < 4; i++) modes[i] = Py_NewRef(m[i]);
    Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(f_##name)), METH_FASTCALL, nullptr}
PyMethodDef functions[] = {{"bind", f_bind, METH_O, nullptr},
                           {"register", f_register, METH_VARARGS, nullptr},
                           FAST(quantized_matmul),
                           FAST(gather_qmm),
                           FAST(qqmm),
                           FAST(quantize),
                           FAST(dequantize),
                           FAST(quantized_embedding),
                           FAST(sorted_offsets),
                           FAST(moe_route),
                           FAST(weighted_sum),
                           FAST(expert_bias_add),
                           FAST(moe_sort),
                           FAST(take_rows),
                           FAST(rms_norm),
                           FAST(add_rms_norm),
                           FAST(swiglu),
                           FAST(quantized_attention),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Arrays and the usual calls of ops.py in C.", -1, functions, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    DeviceType.tp_name = "nuvec_b200._native.DeviceBase";
    DeviceType.tp_basicsize = sizeof(DeviceObject);
    DeviceType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
    DeviceType.tp_new = PyType_GenericNew;
    DeviceType.tp_methods = device_methods;
    ArrayType.tp_name = "nuvec_b200._native.ArrayBase";
    ArrayType.tp_basicsize = sizeof(ArrayObject);
    ArrayType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
    ArrayType.tp_new = PyType_GenericNew;
    ArrayType.tp_init = array_init_py;
    ArrayType.tp_dealloc = array_dealloc;
    ArrayType.tp_methods = array_methods;
    ArrayType.tp_members = array_members;
    ArrayType.tp_getset = array_getset;
    static PyMappingMethods mapping = {nullptr, array_getitem, nullptr};
    ArrayType.tp_as_mapping = &mapping;
    if (PyType_Ready(&DeviceType) < 0 || PyType_Ready(&ArrayType) < 0) return nullptr;
    struct { PyObject **at; const char *text; } const names[] = {{&s_weight, "weight"}, {&s_scales, "scales"}, {&s_biases, "biases"}, {&s_quant, "quant"},
                                                                 {&s_global, "global_scale"}, {&s_mode, "mode"}, {&s_group, "group_size"}, {&s_bits, "bits"},
                                                                 {&s_ptr, "ptr"}, {&s_value, "value"}};
    for (const auto &s : names)
        if (!(*s.at = PyUnicode_InternFromString(s.text))) return nullptr;
    PyObject *m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    if (PyModule_AddObjectRef(m, "DeviceBase", reinterpret_cast<PyObject *>(&DeviceType)) < 0 ||
        PyModule_AddObjectRef(m, "ArrayBase", reinterpret_cast<PyObject *>(&ArrayType)) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
