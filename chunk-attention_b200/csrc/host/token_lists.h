// Conversion of Python lists of token ids.  pybind11's list caster walks a list through the sequence protocol with a
// caster per element.  A prompt is converted twice a step (the cache's and the spans' list), in front of kernels that take 0.17 ms for
// 8192 tokens; the spans' part, its arrays filled, took 157 us for them and takes 49.  Exact lists and tuples of exact ints are read
// directly here; everything else, errors included, is left to the list caster.
//
// Include it in every file that binds functions taking std::vector<int>, so that all agree on the caster.
#pragma once
#include <Python.h>
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <climits>
#include <vector>

namespace pybind11 {
namespace detail {

template <> struct type_caster<std::vector<int>> : list_caster<std::vector<int>, int> {
    bool load(handle src, bool convert) {
        PyObject* o = src.ptr();
        const bool list = PyList_CheckExact(o);
        if (list || PyTuple_CheckExact(o)) {
            const Py_ssize_t n = list ? PyList_GET_SIZE(o) : PyTuple_GET_SIZE(o);
            value.resize((size_t)n);
            Py_ssize_t i = 0;
            for (; i < n; i++) {  // no Python code runs in here: the list keeps its length and its items
                PyObject* x = list ? PyList_GET_ITEM(o, i) : PyTuple_GET_ITEM(o, i);
                if (!PyLong_CheckExact(x)) break;
                int overflow = 0;
                const long v = PyLong_AsLongAndOverflow(x, &overflow);
                if (overflow || v < INT_MIN || v > INT_MAX) break;
                value[(size_t)i] = (int)v;
            }
            if (i == n) return true;
            value.clear();
        }
        return list_caster<std::vector<int>, int>::load(src, convert);
    }
};

}  // namespace detail
}  // namespace pybind11
