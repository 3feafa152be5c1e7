// Python lists to C arrays: token ids, and the entries of a ragged step together with the call (llama_cpp/engine.py loads this with
// ctypes.PyDLL; g++, no CUDA). array.array takes 30 ns a token (2048 of them: 60 us, a tenth of a short prompt's time) and a step's lists of
// slots, lengths, tokens, rows and flags cost 36 us for 32 sequences; here 2 and 3 us.
// Only exact lists and tuples of ints that fit are taken; everything else is left to the caller's general path, which decides what it is.
#include <Python.h>
#include <stdint.h>

#include <new>
#include <vector>

namespace {

inline bool is_seq(PyObject* o) { return PyList_CheckExact(o) || PyTuple_CheckExact(o); }
inline Py_ssize_t len(PyObject* o) { return PySequence_Fast_GET_SIZE(o); }
inline PyObject* at(PyObject* o, Py_ssize_t i) { return PySequence_Fast_GET_ITEM(o, i); }

inline bool to_int32(PyObject* o, int32_t* out) {
    if (!PyLong_Check(o)) return false;
    int over = 0;
    const long v = PyLong_AsLongAndOverflow(o, &over);
    if (over || v < INT32_MIN || v > INT32_MAX) return false;
    *out = (int32_t)v;
    return true;
}

typedef int (*StepFn)(void* engine, int n_entries, const int32_t* slots, const int32_t* n_tokens, const int32_t* tokens, const int32_t* want_rows, int n_want,
                      float* logits, const int32_t* sample, int32_t* sampled);

}  // namespace

// n ints of a list or tuple; 0: it holds something else
extern "C" int b2_py_int32s(PyObject* values, int32_t* out, Py_ssize_t n) {
    if (!is_seq(values) || len(values) != n) return 0;
    for (Py_ssize_t i = 0; i < n; i++) if (!to_int32(at(values, i), out + i)) return 0;
    return 1;
}

static PyObject* step_of_lists(void* step, void* engine, PyObject* entries, PyObject* want, PyObject* sample, int max_entries, int max_tokens, float* logits, int n_want);
// One native step of entries [(slot, [token, ...]), ...] with the rows `want` (or None) and flags `sample` (or None): the list of sampled tokens (None
// where none was asked for), b2_step's code if that is not 0, or None if these are not the plain lists of one step
extern "C" PyObject* b2_py_step(void* step, void* engine, PyObject* entries, PyObject* want, PyObject* sample, int max_entries, int max_tokens, float* logits, int n_want) {
    try {
        return step_of_lists(step, engine, entries, want, sample, max_entries, max_tokens, logits, n_want);
    } catch (const std::bad_alloc&) {
        return PyErr_NoMemory();
    }
}

static PyObject* step_of_lists(void* step, void* engine, PyObject* entries, PyObject* want, PyObject* sample, int max_entries, int max_tokens, float* logits, int n_want) {
    if (!is_seq(entries) || (want != Py_None && !is_seq(want)) || (sample != Py_None && !is_seq(sample))) Py_RETURN_NONE;
    const Py_ssize_t n = len(entries);
    if (n <= 0 || n > max_entries || (want != Py_None && len(want) != n) || (sample != Py_None && len(sample) != n)) Py_RETURN_NONE;
    std::vector<int32_t> slots(n), counts(n), flags(n), sampled(n), tokens, rows;
    for (Py_ssize_t i = 0; i < n; i++) {
        PyObject* e = at(entries, i);
        if (!is_seq(e) || len(e) != 2 || !to_int32(at(e, 0), &slots[i])) Py_RETURN_NONE;
        PyObject* toks = at(e, 1);
        if (!is_seq(toks)) Py_RETURN_NONE;
        const Py_ssize_t k = len(toks), t0 = (Py_ssize_t)tokens.size();
        if (k <= 0 || t0 + k > max_tokens) Py_RETURN_NONE;
        tokens.resize(t0 + k);
        for (Py_ssize_t j = 0; j < k; j++) if (!to_int32(at(toks, j), &tokens[t0 + j])) Py_RETURN_NONE;
        counts[i] = (int32_t)k;
        if (want != Py_None) {
            PyObject* w = at(want, i);
            if (!is_seq(w)) Py_RETURN_NONE;
            for (Py_ssize_t j = 0; j < len(w); j++) {
                int32_t r;
                if (!to_int32(at(w, j), &r) || r < 0 || r >= k) Py_RETURN_NONE;
                rows.push_back((int32_t)(t0 + r));
            }
        }
        if (sample != Py_None) {
            PyObject* f = at(sample, i);
            if (f != Py_True && f != Py_False) Py_RETURN_NONE;
            flags[i] = f == Py_True;
        }
    }
    if ((Py_ssize_t)rows.size() != n_want) Py_RETURN_NONE;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = ((StepFn)step)(engine, (int)n, slots.data(), counts.data(), tokens.data(), n_want ? rows.data() : nullptr, n_want, n_want ? logits : nullptr, flags.data(), sampled.data());
    Py_END_ALLOW_THREADS
    if (rc != 0) return PyLong_FromLong(rc);
    PyObject* out = PyList_New(n);
    for (Py_ssize_t i = 0; out && i < n; i++) {
        PyObject* v = flags[i] ? PyLong_FromLong(sampled[i]) : Py_NewRef(Py_None);
        if (!v) { Py_DECREF(out); return nullptr; }
        PyList_SET_ITEM(out, i, v);
    }
    return out;
}
