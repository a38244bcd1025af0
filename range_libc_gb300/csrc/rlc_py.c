/* _rlcfast -- CPython entry points for the per-call methods of
 * range_libc_gb300.range_libc (the role the reference's Cython module plays).
 *
 * Each function takes a method handle (as an integer) and numpy arrays or
 * CUDA tensors, checks them (arrays through the buffer protocol, tensors
 * through their own attributes) and calls the C ABI directly, tensors on the
 * first one's current stream.  It returns the C ABI status, or -1 when the
 * arguments are not all C-contiguous buffers, or all contiguous CUDA tensors,
 * of the expected item type, rank and length, in which case the Python layer
 * repeats the call through its own argument checks (which raise the
 * reference's errors).  Nothing here computes a range.
 *
 * A call on small tensors is bound by the host: 9.2 us of argument checks,
 * stream lookup and ctypes before, 3.4 us through here.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "rangelibc.h"

#include <string.h>

/* a C-contiguous buffer of `fmt` items ("f" float32, "d" float64) of rank `ndim` */
static int get_buf(PyObject* o, Py_buffer* v, const char* fmt, int ndim, int writable) {
    int flags = PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | (writable ? PyBUF_WRITABLE : 0);
    if (PyObject_GetBuffer(o, v, flags) != 0) {
        PyErr_Clear();
        return -1;
    }
    const char* f = v->format ? v->format : "B";
    if (f[0] == '=' || f[0] == '<' || f[0] == '@') ++f;   /* native little-endian */
    if (strcmp(f, fmt) != 0 || v->ndim != ndim) {
        PyBuffer_Release(v);
        return -1;
    }
    return 0;
}

/* torch's tensor type, its two item types and its current-stream query; looked up once torch is there */
static PyObject *t_tensor, *t_float32, *t_float64, *t_raw_stream;
static PyObject *n_is_cuda, *n_dtype, *n_shape, *n_is_contiguous, *n_data_ptr, *n_get_device;

static int torch_ready(void) {
    if (t_raw_stream) return 1;
    PyObject* name = PyUnicode_FromString("torch");
    PyObject* torch = name ? PyImport_GetModule(name) : NULL;   /* not imported: no argument is a tensor */
    Py_XDECREF(name);
    if (torch) {
        PyObject* c = PyObject_GetAttrString(torch, "_C");
        PyObject* stream = c ? PyObject_GetAttrString(c, "_cuda_getCurrentRawStream") : NULL;
        PyObject* tensor = PyObject_GetAttrString(torch, "Tensor");
        PyObject* f32 = PyObject_GetAttrString(torch, "float32");
        PyObject* f64 = PyObject_GetAttrString(torch, "float64");
        Py_XDECREF(c);
        if (stream && tensor && f32 && f64) {
            t_tensor = tensor;
            t_float32 = f32;
            t_float64 = f64;
            t_raw_stream = stream;
        } else {
            Py_XDECREF(stream);
            Py_XDECREF(tensor);
            Py_XDECREF(f32);
            Py_XDECREF(f64);
        }
        Py_DECREF(torch);
    }
    PyErr_Clear();
    return t_raw_stream != NULL;
}

static int attr_is(PyObject* o, PyObject* name, PyObject* value) {
    PyObject* a = PyObject_GetAttr(o, name);
    const int same = a == value;
    Py_XDECREF(a);
    return same;
}

/* a contiguous CUDA tensor of `fmt` items of rank `ndim` (a plain torch.Tensor: no subclass) */
static int get_dev(PyObject* o, const char* fmt, int ndim, void** ptr, Py_ssize_t* shape) {
    if ((PyObject*)Py_TYPE(o) != t_tensor) return -1;
    if (!attr_is(o, n_is_cuda, Py_True) || !attr_is(o, n_dtype, fmt[0] == 'd' ? t_float64 : t_float32)) goto no;
    PyObject* sh = PyObject_GetAttr(o, n_shape);
    int ok = sh && PyTuple_Check(sh) && PyTuple_GET_SIZE(sh) == ndim;
    for (int i = 0; ok && i < ndim; ++i) {
        shape[i] = PyLong_AsSsize_t(PyTuple_GET_ITEM(sh, i));
        ok = !(shape[i] == -1 && PyErr_Occurred());
    }
    Py_XDECREF(sh);
    if (!ok) goto no;
    PyObject* c = PyObject_CallMethodNoArgs(o, n_is_contiguous);
    ok = c == Py_True;
    Py_XDECREF(c);
    if (!ok) goto no;
    PyObject* p = PyObject_CallMethodNoArgs(o, n_data_ptr);
    if (!p) goto no;
    *ptr = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    if (PyErr_Occurred()) goto no;
    return 0;
no:
    PyErr_Clear();
    return -1;
}

/* the current stream of the tensor's device */
static int get_stream(PyObject* o, void** stream) {
    PyObject* dev = PyObject_CallMethodNoArgs(o, n_get_device);
    PyObject* st = dev ? PyObject_CallOneArg(t_raw_stream, dev) : NULL;
    Py_XDECREF(dev);
    if (st) *stream = PyLong_AsVoidPtr(st);
    Py_XDECREF(st);
    if (!st || PyErr_Occurred()) {
        PyErr_Clear();
        return -1;
    }
    return 0;
}

/* whether the call is one on tensors: then the buffer protocol is not asked */
static int on_device(PyObject* first) { return !PyObject_CheckBuffer(first) && torch_ready(); }

static PyObject* fused(PyObject* self, PyObject* args) {
    (void)self;
    unsigned long long h;
    PyObject *oi, *oa, *oo, *ow;
    if (!PyArg_ParseTuple(args, "KOOOO", &h, &oi, &oa, &oo, &ow)) return NULL;
    if (on_device(oi)) {
        void *pi, *pa, *po, *pw, *st;
        Py_ssize_t si[2], sa[1], so[1], sw[1];
        if (get_dev(oi, "f", 2, &pi, si) || get_dev(oa, "f", 1, &pa, sa) || get_dev(oo, "f", 1, &po, so) ||
            get_dev(ow, "d", 1, &pw, sw) || si[1] != 3 || so[0] < sa[0] || sw[0] < si[0] || si[0] > 0x7fffffff ||
            sa[0] > 0x7fffffff || get_stream(oi, &st))
            return PyLong_FromLong(-1);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_repeat_angles_eval_sensor_model((rlc_method*)(uintptr_t)h, (const float*)pi, (const float*)pa,
                                                             (const float*)po, (double*)pw, (int)si[0], (int)sa[0],
                                                             RLC_DEVICE_PTRS, st);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    Py_buffer bi, ba, bo, bw;
    if (get_buf(oi, &bi, "f", 2, 0)) return PyLong_FromLong(-1);
    if (get_buf(oa, &ba, "f", 1, 0)) { PyBuffer_Release(&bi); return PyLong_FromLong(-1); }
    if (get_buf(oo, &bo, "f", 1, 0)) { PyBuffer_Release(&bi); PyBuffer_Release(&ba); return PyLong_FromLong(-1); }
    if (get_buf(ow, &bw, "d", 1, 1)) {
        PyBuffer_Release(&bi); PyBuffer_Release(&ba); PyBuffer_Release(&bo);
        return PyLong_FromLong(-1);
    }
    int rc = -1;
    const Py_ssize_t n = bi.shape[0], na = ba.shape[0];
    if (bi.shape[1] == 3 && bo.shape[0] >= na && bw.shape[0] >= n && n <= 0x7fffffff && na <= 0x7fffffff) {
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_repeat_angles_eval_sensor_model((rlc_method*)(uintptr_t)h, (const float*)bi.buf,
                                                             (const float*)ba.buf, (const float*)bo.buf,
                                                             (double*)bw.buf, (int)n, (int)na, 0, NULL);
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&bi); PyBuffer_Release(&ba); PyBuffer_Release(&bo); PyBuffer_Release(&bw);
    return PyLong_FromLong(rc);
}

static PyObject* repeat_angles(PyObject* self, PyObject* args) {
    (void)self;
    unsigned long long h;
    PyObject *oi, *oa, *oo;
    if (!PyArg_ParseTuple(args, "KOOO", &h, &oi, &oa, &oo)) return NULL;
    if (on_device(oi)) {
        void *pi, *pa, *po, *st;
        Py_ssize_t si[2], sa[1], so[1];
        if (get_dev(oi, "f", 2, &pi, si) || get_dev(oa, "f", 1, &pa, sa) || get_dev(oo, "f", 1, &po, so) || si[1] != 3 ||
            si[0] > 0x7fffffff || sa[0] > 0x7fffffff || so[0] < si[0] * sa[0] || get_stream(oi, &st))
            return PyLong_FromLong(-1);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_repeat_angles((rlc_method*)(uintptr_t)h, (const float*)pi, (const float*)pa, (float*)po,
                                          (int)si[0], (int)sa[0], RLC_DEVICE_PTRS, st);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    Py_buffer bi, ba, bo;
    if (get_buf(oi, &bi, "f", 2, 0)) return PyLong_FromLong(-1);
    if (get_buf(oa, &ba, "f", 1, 0)) { PyBuffer_Release(&bi); return PyLong_FromLong(-1); }
    if (get_buf(oo, &bo, "f", 1, 1)) { PyBuffer_Release(&bi); PyBuffer_Release(&ba); return PyLong_FromLong(-1); }
    int rc = -1;
    const Py_ssize_t n = bi.shape[0], na = ba.shape[0];
    if (bi.shape[1] == 3 && bo.shape[0] >= n * na && n <= 0x7fffffff && na <= 0x7fffffff) {
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_repeat_angles((rlc_method*)(uintptr_t)h, (const float*)bi.buf, (const float*)ba.buf,
                                          (float*)bo.buf, (int)n, (int)na, 0, NULL);
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&bi); PyBuffer_Release(&ba); PyBuffer_Release(&bo);
    return PyLong_FromLong(rc);
}

static PyObject* calc_range_many(PyObject* self, PyObject* args) {
    (void)self;
    unsigned long long h;
    PyObject *oi, *oo;
    if (!PyArg_ParseTuple(args, "KOO", &h, &oi, &oo)) return NULL;
    if (on_device(oi)) {
        void *pi, *po, *st;
        Py_ssize_t si[2], so[1];
        if (get_dev(oi, "f", 2, &pi, si) || get_dev(oo, "f", 1, &po, so) || si[1] != 3 || si[0] < so[0] ||
            so[0] > 0x7fffffff || get_stream(oi, &st))
            return PyLong_FromLong(-1);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_many((rlc_method*)(uintptr_t)h, (const float*)pi, (float*)po, (int)so[0], RLC_DEVICE_PTRS, st);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    Py_buffer bi, bo;
    if (get_buf(oi, &bi, "f", 2, 0)) return PyLong_FromLong(-1);
    if (get_buf(oo, &bo, "f", 1, 1)) { PyBuffer_Release(&bi); return PyLong_FromLong(-1); }
    int rc = -1;
    const Py_ssize_t n = bo.shape[0];   /* the reference takes the count from outs */
    if (bi.shape[1] == 3 && bi.shape[0] >= n && n <= 0x7fffffff) {
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_calc_range_many((rlc_method*)(uintptr_t)h, (const float*)bi.buf, (float*)bo.buf, (int)n, 0, NULL);
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&bi); PyBuffer_Release(&bo);
    return PyLong_FromLong(rc);
}

static PyObject* eval_sensor_model(PyObject* self, PyObject* args) {
    (void)self;
    unsigned long long h;
    PyObject *oo, *orr, *ow;
    int nr, np_;
    if (!PyArg_ParseTuple(args, "KOOOii", &h, &oo, &orr, &ow, &nr, &np_)) return NULL;
    if (on_device(oo)) {
        void *po, *pr, *pw, *st;
        Py_ssize_t so[1], sr[1], sw[1];
        if (get_dev(oo, "f", 1, &po, so) || get_dev(orr, "f", 1, &pr, sr) || get_dev(ow, "d", 1, &pw, sw) || nr < 0 ||
            np_ < 0 || so[0] < nr || sr[0] < (Py_ssize_t)nr * np_ || sw[0] < np_ || get_stream(oo, &st))
            return PyLong_FromLong(-1);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_eval_sensor_model((rlc_method*)(uintptr_t)h, (const float*)po, (const float*)pr, (double*)pw, nr, np_,
                                   RLC_DEVICE_PTRS, st);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(rc);
    }
    Py_buffer bo, br, bw;
    if (get_buf(oo, &bo, "f", 1, 0)) return PyLong_FromLong(-1);
    if (get_buf(orr, &br, "f", 1, 0)) { PyBuffer_Release(&bo); return PyLong_FromLong(-1); }
    if (get_buf(ow, &bw, "d", 1, 1)) { PyBuffer_Release(&bo); PyBuffer_Release(&br); return PyLong_FromLong(-1); }
    int rc = -1;
    if (nr >= 0 && np_ >= 0 && bo.shape[0] >= nr && br.shape[0] >= (Py_ssize_t)nr * np_ && bw.shape[0] >= np_) {
        Py_BEGIN_ALLOW_THREADS
        rc = rlc_eval_sensor_model((rlc_method*)(uintptr_t)h, (const float*)bo.buf, (const float*)br.buf,
                                   (double*)bw.buf, nr, np_, 0, NULL);
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&bo); PyBuffer_Release(&br); PyBuffer_Release(&bw);
    return PyLong_FromLong(rc);
}

static PyMethodDef kMethods[] = {
    {"fused", fused, METH_VARARGS, "calc_range_repeat_angles_eval_sensor_model"},
    {"repeat_angles", repeat_angles, METH_VARARGS, "calc_range_repeat_angles"},
    {"calc_range_many", calc_range_many, METH_VARARGS, "calc_range_many"},
    {"eval_sensor_model", eval_sensor_model, METH_VARARGS, "eval_sensor_model"},
    {NULL, NULL, 0, NULL},
};

static struct PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_rlcfast", NULL, -1, kMethods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__rlcfast(void) {
    n_is_cuda = PyUnicode_InternFromString("is_cuda");
    n_dtype = PyUnicode_InternFromString("dtype");
    n_shape = PyUnicode_InternFromString("shape");
    n_is_contiguous = PyUnicode_InternFromString("is_contiguous");
    n_data_ptr = PyUnicode_InternFromString("data_ptr");
    n_get_device = PyUnicode_InternFromString("get_device");
    if (!n_is_cuda || !n_dtype || !n_shape || !n_is_contiguous || !n_data_ptr || !n_get_device) return NULL;
    return PyModule_Create(&kModule);
}
