/*
 * Packers of the Python binding: gate lists and Hamiltonians as the C ABI's
 * arrays.  A gate list of Python tuples is walked once through the CPython
 * API (3,000 gates: 0.6 ms in Python, most of a small circuit's call).
 *
 * Every function returns a negative value, with no Python error set, for
 * anything but plain tuples and lists of numbers in range; the caller then
 * takes its Python path, which accepts more and raises what it always raised.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <string.h>

typedef struct {
    uint32_t kind, target;
    uint64_t control_mask;
    double angle;
} gate_t;

static int small_int(PyObject *o, long limit, long *out) {
    long v;
    if (!PyLong_CheckExact(o)) return -1;
    v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return -1;
    }
    if (v < 0 || v >= limit) return -1;
    *out = v;
    return 0;
}

static int number(PyObject *o, double *out) {
    if (PyFloat_CheckExact(o)) {
        *out = PyFloat_AS_DOUBLE(o);
        return 0;
    }
    if (PyLong_CheckExact(o)) {
        *out = PyLong_AsDouble(o);
        if (*out == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            return -1;
        }
        return 0;
    }
    return -1;
}

#define IS_SEQ(o) (PyTuple_CheckExact(o) || PyList_CheckExact(o))

/* circuit: list or tuple of (kind, target, controls, angle); n records. */
long kbwg_pack_gates(PyObject *circuit, gate_t *out, long n) {
    long i, j, v;
    PyObject **items;
    if (!IS_SEQ(circuit) || PySequence_Fast_GET_SIZE(circuit) != n) return -1;
    items = PySequence_Fast_ITEMS(circuit);
    for (i = 0; i < n; i++) {
        PyObject *g = items[i], **f, *c, **cs;
        Py_ssize_t nc;
        if (!IS_SEQ(g) || PySequence_Fast_GET_SIZE(g) != 4) return -1;
        f = PySequence_Fast_ITEMS(g);
        if (small_int(f[0], 1L << 31, &v)) return -1;
        out[i].kind = (uint32_t)v;
        if (small_int(f[1], 1L << 31, &v)) return -1;
        out[i].target = (uint32_t)v;
        c = f[2];
        if (!IS_SEQ(c)) return -1;
        nc = PySequence_Fast_GET_SIZE(c);
        cs = PySequence_Fast_ITEMS(c);
        out[i].control_mask = 0;
        for (j = 0; j < nc; j++) {
            if (small_int(cs[j], 64, &v) || (out[i].control_mask >> v & 1)) return -1;
            out[i].control_mask |= 1ull << v;
        }
        if (number(f[3], &out[i].angle)) return -1;
    }
    return 0;
}

/* Number of (pauli, qubit) terms of a Hamiltonian [(coefficient, [(pauli, qubit), ...]), ...]. */
long kbwg_count_terms(PyObject *ham, long n) {
    long i, total = 0;
    PyObject **items;
    if (!IS_SEQ(ham) || PySequence_Fast_GET_SIZE(ham) != n) return -1;
    items = PySequence_Fast_ITEMS(ham);
    for (i = 0; i < n; i++) {
        PyObject **f;
        if (!IS_SEQ(items[i]) || PySequence_Fast_GET_SIZE(items[i]) != 2) return -1;
        f = PySequence_Fast_ITEMS(items[i]);
        if (!IS_SEQ(f[1])) return -1;
        total += (long)PySequence_Fast_GET_SIZE(f[1]);
    }
    return total;
}

/* paulis, qubits: kbwg_count_terms() entries; offsets: n + 1; coefs: n. */
long kbwg_pack_terms(PyObject *ham, long n, long total, uint8_t *paulis, uintptr_t *qubits, uintptr_t *offsets,
                     double *coefs) {
    long i, k = 0, v;
    Py_ssize_t j;
    PyObject **items;
    if (!IS_SEQ(ham) || PySequence_Fast_GET_SIZE(ham) != n) return -1;
    items = PySequence_Fast_ITEMS(ham);
    offsets[0] = 0;
    for (i = 0; i < n; i++) {
        PyObject **f = PySequence_Fast_ITEMS(items[i]), **t;
        Py_ssize_t nt = PySequence_Fast_GET_SIZE(f[1]);
        if (number(f[0], &coefs[i])) return -1;
        t = PySequence_Fast_ITEMS(f[1]);
        for (j = 0; j < nt; j++) {
            PyObject **pq;
            if (k >= total || !IS_SEQ(t[j]) || PySequence_Fast_GET_SIZE(t[j]) != 2) return -1;
            pq = PySequence_Fast_ITEMS(t[j]);
            if (small_int(pq[0], 256, &v)) return -1;
            paulis[k] = (uint8_t)v;
            if (small_int(pq[1], 1L << 31, &v)) return -1;
            qubits[k] = (uintptr_t)v;
            k++;
        }
        offsets[i + 1] = (uintptr_t)k;
    }
    return k == total ? 0 : -1;
}
