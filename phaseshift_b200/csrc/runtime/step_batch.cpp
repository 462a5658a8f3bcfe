// Expansion of a step's requests into the packed arrays that the kernels index (runtime/batch.py: StepBatch): with array operations or
// a loop in Python it cost 6 to 15 us of host time per sequence, between two steps with nothing for the GPU to do: 32 sequences of one
// row 468 us, 32 us here on the same host.
#include <cstring>
#include <stdexcept>
#include <string>

#include <pybind11/pybind11.h>

#include "ps_sampling.h"

namespace py = pybind11;

namespace {

// Field `name` of a request; the name object lives as long as the module.
struct Name {
    PyObject* s;
    explicit Name(const char* n) : s(PyUnicode_InternFromString(n)) {}
    py::object of(PyObject* o) const {
        PyObject* v = PyObject_GetAttr(o, s);
        if (v == nullptr) throw py::error_already_set();
        return py::reinterpret_steal<py::object>(v);
    }
};

// A Python integer for `o`, as an assignment to an element of an integer array takes it: integers of any type, floats and texts (cut and
// read by int()), but no arrays.  `wraps`: numpy's and torch's own integers keep their low bits, where Python's have to fit.
py::object as_integer(PyObject* o, bool& wraps) {
    wraps = !PyLong_Check(o);
    PyObject* i = PyNumber_Index(o);
    if (i == nullptr && (PyFloat_Check(o) || PyUnicode_Check(o) || !PySequence_Check(o)) && PyErr_ExceptionMatches(PyExc_TypeError)) {
        PyErr_Clear();
        wraps = false;
        i = PyNumber_Long(o);
        if (i == nullptr && PyUnicode_Check(o) && PyErr_ExceptionMatches(PyExc_ValueError)) {
            PyErr_Clear();
            throw py::type_error("a number is needed");
        }
    }
    if (i == nullptr) throw py::error_already_set();
    return py::reinterpret_steal<py::object>(i);
}
int32_t fit_i32(PyObject* i, const char* what) {
    const long long v = PyLong_AsLongLong(i);
    if (v == -1 && PyErr_Occurred()) throw py::error_already_set();
    if (v < INT32_MIN || v > INT32_MAX) throw std::overflow_error(std::string(what) + " does not fit 32 bits");
    return (int32_t)v;
}
int32_t to_i32(PyObject* o, const char* what) {
    if (PyLong_CheckExact(o)) return fit_i32(o, what);
    bool wraps;
    const py::object i = as_integer(o, wraps);
    return wraps ? (int32_t)(uint32_t)PyLong_AsUnsignedLongLongMask(i.ptr()) : fit_i32(i.ptr(), what);
}
uint64_t to_u64(PyObject* o) {
    bool wraps;
    const py::object i = as_integer(o, wraps);
    if (wraps) return PyLong_AsUnsignedLongLongMask(i.ptr());
    const unsigned long long v = PyLong_AsUnsignedLongLong(i.ptr());
    if (v == (unsigned long long)-1 && PyErr_Occurred()) throw py::error_already_set();
    return v;
}
uint32_t to_u32(PyObject* o, const char* what) {
    bool wraps;
    const py::object i = as_integer(o, wraps);
    if (wraps) return (uint32_t)PyLong_AsUnsignedLongLongMask(i.ptr());
    const long long v = PyLong_AsLongLong(i.ptr());
    if (v == -1 && PyErr_Occurred()) throw py::error_already_set();
    if (v < 0 || v > UINT32_MAX) throw std::overflow_error(std::string(what) + " does not fit 32 bits");
    return (uint32_t)v;
}
double to_double(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw py::error_already_set();
    return v;
}

// A request's sequence as a list or tuple.
struct Items {
    PyObject* fast;
    explicit Items(const py::object& o) : fast(PySequence_Fast(o.ptr(), "token_ids and output_rows are sequences")) {
        if (fast == nullptr) throw py::error_already_set();
    }
    ~Items() { Py_DECREF(fast); }
    Items(const Items&) = delete;
    Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(fast); }
    PyObject* operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(fast, i); }
};

// A sequence's token ids are one row of numbers: a list, a tuple, a range, an array or a tensor of one dimension.
void check_row(const py::object& o) {
    if (PyList_CheckExact(o.ptr()) || PyTuple_CheckExact(o.ptr())) return;
    if (PyBytes_Check(o.ptr()) || PyUnicode_Check(o.ptr())) throw py::value_error("token_ids are numbers");
    if (PyAnySet_Check(o.ptr()) || PyDict_Check(o.ptr())) throw py::type_error("token_ids is a sequence");
    if (PyObject_Size(o.ptr()) < 0) throw py::error_already_set();
    if (py::hasattr(o, "ndim") && py::cast<long long>(o.attr("ndim")) != 1) throw py::value_error("token_ids has one dimension");
}

// ints: [ids | row_slot | row_pos] of `max_rows`, [max_seqs][4] descriptors, output rows and short-sequence positions of `max_rows`;
// samp: sampling rows.  Returns (rows, output rows, largest visible length, output row i is step row i for every i).
py::tuple fill_step(uintptr_t ints, uintptr_t samp, int max_rows, int max_seqs, int short_rows, const py::sequence& seqs) {
    static const Name n_slot("slot"), n_pos("pos_start"), n_ids("token_ids"), n_out_rows("output_rows"), n_temp("temperature"), n_top_p("top_p"),
        n_top_k("top_k"), n_seed("seed"), n_index("sample_index");
    int32_t* a = reinterpret_cast<int32_t*>(ints);
    ps::SamplingRow* sp = reinterpret_cast<ps::SamplingRow*>(samp);
    int32_t *ids = a, *slot = a + max_rows, *pos = slot + max_rows, *desc = pos + max_rows, *outs = desc + 4 * (size_t)max_seqs, *pshort = outs + max_rows;
    const Items list(seqs);
    const int n = (int)list.size();
    if (n > max_seqs) throw py::value_error("too many sequences for this batch");
    // padding rows of a bucket: slot -1 / position -1, skipped by the kernels
    std::memset(a, 0, sizeof(int32_t) * (5 * (size_t)max_rows + 4 * (size_t)max_seqs));
    std::memset(slot, 0xff, sizeof(int32_t) * 2 * (size_t)max_rows);
    std::memset(pshort, 0xff, sizeof(int32_t) * (size_t)max_rows);
    int r = 0, n_out = 0;
    long long visible = 1;
    bool identity = true;
    for (int i = 0; i < n; ++i) {
        PyObject* s = list[i];
        const py::object given = n_ids.of(s);
        check_row(given);
        const Items tok(given);
        const int k = (int)tok.size();
        if (k > max_rows - r) throw py::value_error("too many rows for this batch");
        const int32_t sl = to_i32(n_slot.of(s).ptr(), "slot"), p0 = to_i32(n_pos.of(s).ptr(), "pos_start");
        if ((long long)p0 + k - 1 > INT32_MAX) throw std::overflow_error("pos_start does not fit 32 bits");
        for (int j = 0; j < k; ++j) {
            ids[r + j] = to_i32(tok[j], "token id");
            slot[r + j] = sl;
            pos[r + j] = p0 + j;
            pshort[r + j] = k <= short_rows ? p0 + j : -2;
        }
        int32_t* d = desc + 4 * i;
        d[0] = r; d[1] = k; d[2] = sl; d[3] = p0;
        const Items rows(n_out_rows.of(s));
        if (rows.size() > max_rows - n_out) throw py::value_error("too many output rows for this batch");
        if (rows.size() > 0) {
            ps::SamplingRow row;
            const double t = to_double(n_temp.of(s).ptr());
            row.mode = t <= 0.0 ? ps::kSamplingGreedy : ps::kSamplingStochastic;
            row.temperature = (float)t;
            row.top_p = (float)to_double(n_top_p.of(s).ptr());
            row.top_k = to_u32(n_top_k.of(s).ptr(), "top_k");
            row.seed = to_u64(n_seed.of(s).ptr());
            row.sample_index = to_u64(n_index.of(s).ptr());
            if (row.sample_index + (uint64_t)(rows.size() - 1) < row.sample_index) throw std::overflow_error("sample_index does not fit 64 bits");
            for (Py_ssize_t j = 0; j < rows.size(); ++j, ++n_out) {
                outs[n_out] = r + to_i32(rows[j], "output row");
                identity = identity && outs[n_out] == n_out;
                sp[n_out] = row;
                ++row.sample_index;
            }
        }
        if (p0 + (long long)k > visible) visible = p0 + (long long)k;
        r += k;
    }
    return py::make_tuple(r, n_out, visible, identity && n_out == r);
}

}  // namespace

void bind_step_batch(py::module_& m) {
    m.def("fill_step", &fill_step, py::arg("ints"), py::arg("samp"), py::arg("max_rows"), py::arg("max_seqs"), py::arg("short_rows"), py::arg("seqs"));
}
