// Host-side packing of a batch of requests (CPython extension module _xr_host).
//
// fill(items, type_map, types_out, x_out) walks the batch's request tuples
// (symbols, positions, total_charge, cell, pbc, initial_charges) once in C: each symbol is looked up in
// type_map (label -> type index) and written to types_out (int32, the batch's atoms in order), and
// positions that are a C-contiguous float64 (n, 3) buffer are copied into x_out (float64, atoms x 3)
// after a finiteness check. A request this cannot take as is (another container or dtype, a label
// missing from the map, a non-finite coordinate, a total charge that is not a finite int or float)
// is left for the Python path, which applies xreac's validation and messages; fill returns the
// indices of those requests.
//
// guesses(items, addr_out) takes the requests' initial charges: None gives address 0, a C-contiguous
// float64 numpy array of one finite charge per atom gives its data address (valid while the caller
// holds the request; other buffer exporters may not keep their memory after the export ends), and
// anything else is left for the Python checks; it returns the indices of those.
//
// items(systems) makes the request tuples of evaluate_many's keyword dicts; cells(items, cutoff,
// max_expanded_atoms, block) takes fully periodic cells given as float64 arrays, with the scalar arithmetic
// of geometry.periodic_cell; evaluations(...) makes a batch's result objects and field(evaluation, name)
// one of their array fields on its first access (the views of _BatchResults.field). In Python these
// took 0.65 of the 1.8 ms of a batch of 192 small requests whose results are read.
#include <Python.h>

#include <cmath>
#include <cstring>

namespace {

bool finite_number(PyObject* q) {
  if (PyFloat_CheckExact(q)) return std::isfinite(PyFloat_AS_DOUBLE(q));
  return PyLong_CheckExact(q) != 0;
}

// 0: taken; 1: left for Python; -1: a Python error is set
int fill_one(PyObject* item, PyObject* type_map, int* types, double* x, Py_ssize_t natoms) {
  if (!PyTuple_Check(item) || PyTuple_GET_SIZE(item) != 6) return 1;
  PyObject* symbols = PyTuple_GET_ITEM(item, 0);
  PyObject* positions = PyTuple_GET_ITEM(item, 1);
  if (!finite_number(PyTuple_GET_ITEM(item, 2))) return 1;
  if (!PyList_CheckExact(symbols) && !PyTuple_CheckExact(symbols)) return 1;
  PyObject** sym = PySequence_Fast_ITEMS(symbols);
  if (PySequence_Fast_GET_SIZE(symbols) != natoms || natoms == 0) return 1;
  // Labels repeat, usually as the same string objects: a few recently seen objects are matched by
  // identity before the dictionary is asked.
  constexpr int kSeen = 8;
  PyObject* seen[kSeen] = {};
  int seen_type[kSeen] = {};
  int nseen = 0;
  for (Py_ssize_t a = 0; a < natoms; ++a) {
    PyObject* label = sym[a];
    int k = 0;
    while (k < nseen && seen[k] != label) ++k;
    if (k < nseen) {
      types[a] = seen_type[k];
      continue;
    }
    if (!PyUnicode_CheckExact(label)) return 1;
    PyObject* t = PyDict_GetItemWithError(type_map, label);  // borrowed
    if (!t) return PyErr_Occurred() ? -1 : 1;
    const long v = PyLong_AsLong(t);
    if (v == -1 && PyErr_Occurred()) return -1;
    types[a] = (int)v;
    if (nseen < kSeen) {
      seen[nseen] = label;
      seen_type[nseen++] = (int)v;
    }
  }
  Py_buffer view;
  if (PyObject_GetBuffer(positions, &view, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | PyBUF_ND) != 0) {
    PyErr_Clear();
    return 1;
  }
  int rc = 1;
  if (view.ndim == 2 && view.shape[0] == natoms && view.shape[1] == 3 && view.itemsize == 8 && view.format &&
      std::strcmp(view.format, "d") == 0) {
    const double* src = static_cast<const double*>(view.buf);
    bool ok = true;
    for (Py_ssize_t k = 0; k < 3 * natoms; ++k) ok = ok && std::isfinite(src[k]);
    if (ok) {
      std::memcpy(x, src, sizeof(double) * 3 * (size_t)natoms);
      rc = 0;
    }
  }
  PyBuffer_Release(&view);
  return rc;
}

PyObject* fill(PyObject*, PyObject* args) {
  PyObject *items, *type_map, *types_obj, *x_obj;
  if (!PyArg_ParseTuple(args, "O!O!OO", &PyList_Type, &items, &PyDict_Type, &type_map, &types_obj, &x_obj)) return nullptr;
  Py_buffer tv, xv;
  if (PyObject_GetBuffer(types_obj, &tv, PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE | PyBUF_FORMAT) != 0) return nullptr;
  if (PyObject_GetBuffer(x_obj, &xv, PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE | PyBUF_FORMAT) != 0) {
    PyBuffer_Release(&tv);
    return nullptr;
  }
  PyObject* slow = nullptr;
  const Py_ssize_t total = tv.len / (Py_ssize_t)sizeof(int);
  if (tv.itemsize != 4 || xv.itemsize != 8 || xv.len != 3 * tv.len * 2) {
    PyErr_SetString(PyExc_ValueError, "fill needs int32 types and float64 (atoms, 3) positions");
  } else if ((slow = PyList_New(0)) != nullptr) {
    int* types = static_cast<int*>(tv.buf);
    double* x = static_cast<double*>(xv.buf);
    Py_ssize_t off = 0;
    const Py_ssize_t nitems = PyList_GET_SIZE(items);
    for (Py_ssize_t k = 0; k < nitems; ++k) {
      PyObject* item = PyList_GET_ITEM(items, k);
      if (!PyTuple_Check(item) || PyTuple_GET_SIZE(item) < 1) {
        PyErr_SetString(PyExc_ValueError, "requests must be tuples");
        Py_CLEAR(slow);
        break;
      }
      const Py_ssize_t n = PyObject_Length(PyTuple_GET_ITEM(item, 0));
      if (n < 0 || off + n > total) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "atom counts do not match the output size");
        Py_CLEAR(slow);
        break;
      }
      const int rc = fill_one(item, type_map, types + off, x + 3 * off, n);
      if (rc < 0) {
        Py_CLEAR(slow);
        break;
      }
      if (rc == 1) {
        PyObject* idx = PyLong_FromSsize_t(k);
        if (!idx || PyList_Append(slow, idx) != 0) {
          Py_XDECREF(idx);
          Py_CLEAR(slow);
          break;
        }
        Py_DECREF(idx);
      }
      off += n;
    }
  }
  PyBuffer_Release(&tv);
  PyBuffer_Release(&xv);
  return slow;
}

// 0: taken (address in *addr, 0 for None); 1: left for Python
int guess_one(PyObject* item, unsigned long long* addr) {
  *addr = 0;
  if (!PyTuple_Check(item) || PyTuple_GET_SIZE(item) != 6) return 1;
  PyObject* initial = PyTuple_GET_ITEM(item, 5);
  if (initial == Py_None) return 0;
  if (std::strcmp(Py_TYPE(initial)->tp_name, "numpy.ndarray") != 0) return 1;
  const Py_ssize_t n = PyObject_Length(PyTuple_GET_ITEM(item, 0));
  if (n < 0) {
    PyErr_Clear();
    return 1;
  }
  Py_buffer view;
  if (PyObject_GetBuffer(initial, &view, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | PyBUF_ND) != 0) {
    PyErr_Clear();
    return 1;
  }
  int rc = 1;
  if (view.ndim == 1 && view.shape[0] == n && view.itemsize == 8 && view.format && std::strcmp(view.format, "d") == 0) {
    const double* q = static_cast<const double*>(view.buf);
    bool ok = true;
    for (Py_ssize_t k = 0; k < n; ++k) ok = ok && std::isfinite(q[k]);
    if (ok) {
      *addr = reinterpret_cast<unsigned long long>(view.buf);
      rc = 0;
    }
  }
  PyBuffer_Release(&view);
  return rc;
}

PyObject* guesses(PyObject*, PyObject* args) {
  PyObject *items, *addr_obj;
  if (!PyArg_ParseTuple(args, "O!O", &PyList_Type, &items, &addr_obj)) return nullptr;
  Py_buffer av;
  if (PyObject_GetBuffer(addr_obj, &av, PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE | PyBUF_FORMAT) != 0) return nullptr;
  const Py_ssize_t nitems = PyList_GET_SIZE(items);
  PyObject* slow = nullptr;
  if (av.itemsize != 8 || av.len != 8 * nitems) {
    PyErr_SetString(PyExc_ValueError, "guesses needs one uint64 address per request");
  } else if ((slow = PyList_New(0)) != nullptr) {
    unsigned long long* addr = static_cast<unsigned long long*>(av.buf);
    for (Py_ssize_t k = 0; k < nitems; ++k) {
      if (guess_one(PyList_GET_ITEM(items, k), addr + k) == 0) continue;
      PyObject* idx = PyLong_FromSsize_t(k);
      if (!idx || PyList_Append(slow, idx) != 0) {
        Py_XDECREF(idx);
        Py_CLEAR(slow);
        break;
      }
      Py_DECREF(idx);
    }
  }
  PyBuffer_Release(&av);
  return slow;
}

// The request tuples of a sequence of keyword dicts, or None when it is something else.
PyObject* items(PyObject*, PyObject* systems) {
  if (!PyList_CheckExact(systems) && !PyTuple_CheckExact(systems)) Py_RETURN_NONE;
  static const char* const names[6] = {"symbols", "positions", "total_charge", "cell", "pbc", "initial_charges"};
  static PyObject* key[6];
  static PyObject* zero;
  for (int q = 0; q < 6; ++q)
    if (!key[q] && !(key[q] = PyUnicode_InternFromString(names[q]))) return nullptr;
  if (!zero && !(zero = PyLong_FromLong(0))) return nullptr;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(systems);
  PyObject** in = PySequence_Fast_ITEMS(systems);
  for (Py_ssize_t k = 0; k < n; ++k)
    if (!PyDict_CheckExact(in[k])) Py_RETURN_NONE;
  PyObject* out = PyList_New(n);
  for (Py_ssize_t k = 0; out && k < n; ++k) {
    PyObject* t = PyTuple_New(6);
    if (!t) {
      Py_CLEAR(out);
      break;
    }
    PyList_SET_ITEM(out, k, t);
    for (int q = 0; q < 6; ++q) {
      PyObject* v = PyDict_GetItemWithError(in[k], key[q]);  // borrowed
      if (!v) {
        if (PyErr_Occurred() || q < 2) {
          if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key[q]);
          Py_CLEAR(out);
          break;
        }
        v = q == 2 ? zero : Py_None;
      }
      Py_INCREF(v);
      PyTuple_SET_ITEM(t, q, v);
    }
  }
  return out;
}

// Whether `cell` is a float64 array of three lengths or a matrix that the general path would accept as a
// fully periodic cell, with its matrix and replication counts (geometry.periodic_cell, which see).
bool periodic(PyObject* cell, double cutoff, Py_ssize_t atoms, double limit, double* m, long reps[3]) {
  if (std::strcmp(Py_TYPE(cell)->tp_name, "numpy.ndarray") != 0) return false;
  Py_buffer view;
  if (PyObject_GetBuffer(cell, &view, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT | PyBUF_ND) != 0) {
    PyErr_Clear();
    return false;
  }
  bool ok = view.itemsize == 8 && view.format && std::strcmp(view.format, "d") == 0;
  const double* v = static_cast<const double*>(view.buf);
  if (ok && view.ndim == 1 && view.shape[0] == 3) {
    for (int k = 0; k < 9; ++k) m[k] = k % 4 == 0 ? v[k / 4] : 0.0;
    ok = v[0] > 0 && v[1] > 0 && v[2] > 0;
  } else if (ok && view.ndim == 2 && view.shape[0] == 3 && view.shape[1] == 3) {
    std::memcpy(m, v, 9 * sizeof(double));
  } else {
    ok = false;
  }
  PyBuffer_Release(&view);
  if (!ok) return false;
  for (int k = 0; k < 9; ++k)
    if (!std::isfinite(m[k])) return false;
  const double *a = m, *b = m + 3, *c = m + 6;
  const double face[3][3] = {{b[1] * c[2] - b[2] * c[1], b[2] * c[0] - b[0] * c[2], b[0] * c[1] - b[1] * c[0]},
                             {c[1] * a[2] - c[2] * a[1], c[2] * a[0] - c[0] * a[2], c[0] * a[1] - c[1] * a[0]},
                             {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]}};
  const double det = a[0] * face[0][0] + a[1] * face[0][1] + a[2] * face[0][2];
  double scale = 1e-12;
  for (int r = 0; r < 3; ++r) scale *= std::sqrt(m[3 * r] * m[3 * r] + m[3 * r + 1] * m[3 * r + 1] + m[3 * r + 2] * m[3 * r + 2]);
  if (!(det > scale)) return false;
  double copies = 1.0;
  for (int k = 0; k < 3; ++k) {
    const double* f = face[k];
    const double ratio = cutoff * (1 + 1e-12) * std::sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]) / det;
    if (!(ratio < 1e6) || std::fabs(ratio - std::nearbyint(ratio)) < 1e-9) return false;
    reps[k] = (long)std::floor(ratio) + 1;
    copies *= (double)reps[k];
  }
  return !(copies > 1 && copies * (double)atoms > limit);
}

// ([(index, repetitions)] of the requests whose cells it wrote into their rows of `block` (float64, one 3 x 3
// matrix per request), [index] of the other periodic ones, which are left for Python).
PyObject* cells(PyObject*, PyObject* args) {
  PyObject *list, *block_obj;
  double cutoff, limit;
  if (!PyArg_ParseTuple(args, "O!ddO", &PyList_Type, &list, &cutoff, &limit, &block_obj)) return nullptr;
  Py_buffer bv;
  if (PyObject_GetBuffer(block_obj, &bv, PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE | PyBUF_FORMAT) != 0) return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(list);
  PyObject *fast = PyList_New(0), *slow = PyList_New(0);
  bool ok = fast && slow;
  if (ok && (bv.itemsize != 8 || bv.len != 72 * n)) {
    PyErr_SetString(PyExc_ValueError, "cells needs one float64 3 x 3 matrix per request");
    ok = false;
  }
  for (Py_ssize_t k = 0; ok && k < n; ++k) {
    PyObject* item = PyList_GET_ITEM(list, k);
    if (!PyTuple_Check(item) || PyTuple_GET_SIZE(item) != 6) {
      PyErr_SetString(PyExc_ValueError, "requests must be tuples");
      ok = false;
      break;
    }
    PyObject *cell = PyTuple_GET_ITEM(item, 3), *pbc = PyTuple_GET_ITEM(item, 4);
    if ((pbc == Py_None && cell == Py_None) || pbc == Py_False) continue;
    const Py_ssize_t atoms = PyObject_Length(PyTuple_GET_ITEM(item, 0));
    if (atoms < 0) {
      ok = false;
      break;
    }
    long r[3];
    PyObject* entry;
    const bool taken = (pbc == Py_True || pbc == Py_None) &&
                       periodic(cell, cutoff, atoms, limit, static_cast<double*>(bv.buf) + 9 * k, r);
    entry = taken ? Py_BuildValue("n(lll)", k, r[0], r[1], r[2]) : PyLong_FromSsize_t(k);
    ok = entry && PyList_Append(taken ? fast : slow, entry) == 0;
    Py_XDECREF(entry);
  }
  PyBuffer_Release(&bv);
  if (!ok) {
    Py_XDECREF(fast);
    Py_XDECREF(slow);
    return nullptr;
  }
  return Py_BuildValue("NN", fast, slow);
}

// Interned names of the result objects' fields.
enum { N_BATCH, N_INDEX, N_ENERGY, N_FULL, N_REPS, N_BACKEND, N_FORCES, N_CHARGES, N_TBO, N_NLP, N_COUNTS, N_DIPOLE, N_BONDS,
       N_COMPONENTS, N_OFFSETS, N_CUT, N_NAMES };
const char* const kNames[N_NAMES] = {"_batch", "_index", "energy", "full_derivative", "cell_repetitions", "neighbor_backend",
                                     "forces", "charges", "total_bond_orders", "lone_pairs", "bond_counts", "dipole",
                                     "bonds", "components", "offsets", "cut"};
PyObject* name_of[N_NAMES];

// evaluations(cls, energies, full_derivative, repetitions, backend, batch): one instance of cls per system.
PyObject* evaluations(PyObject*, PyObject* args) {
  PyObject *cls, *energies, *full, *reps, *backend, *batch;
  if (!PyArg_ParseTuple(args, "O!O!OO!OO", &PyType_Type, &cls, &PyList_Type, &energies, &full, &PyList_Type, &reps, &backend,
                        &batch))
    return nullptr;
  const Py_ssize_t n = PyList_GET_SIZE(energies);
  if (PyList_GET_SIZE(reps) != n) {
    PyErr_SetString(PyExc_ValueError, "one entry per system");
    return nullptr;
  }
  PyObject *out = PyList_New(n), *none = PyTuple_New(0);
  for (Py_ssize_t k = 0; out && none && k < n; ++k) {
    PyObject* ev = PyBaseObject_Type.tp_new((PyTypeObject*)cls, none, nullptr);
    PyObject* dict = ev ? PyObject_GenericGetDict(ev, nullptr) : nullptr;
    PyObject* index = PyLong_FromSsize_t(k);
    const bool ok = dict && index && PyDict_SetItem(dict, name_of[N_ENERGY], PyList_GET_ITEM(energies, k)) == 0 &&
                    PyDict_SetItem(dict, name_of[N_FULL], full) == 0 &&
                    PyDict_SetItem(dict, name_of[N_REPS], PyList_GET_ITEM(reps, k)) == 0 &&
                    PyDict_SetItem(dict, name_of[N_BACKEND], backend) == 0 &&
                    PyDict_SetItem(dict, name_of[N_BATCH], batch) == 0 && PyDict_SetItem(dict, name_of[N_INDEX], index) == 0;
    Py_XDECREF(dict);
    Py_XDECREF(index);
    if (!ok) {
      Py_XDECREF(ev);
      Py_CLEAR(out);
      break;
    }
    PyList_SET_ITEM(out, k, ev);
  }
  Py_XDECREF(none);
  return out;
}

// array[beg:end] of an attribute of the batch
PyObject* part(PyObject* array, PyObject* beg, PyObject* end) {
  PyObject* slice = PySlice_New(beg, end, nullptr);
  PyObject* v = slice ? PyObject_GetItem(array, slice) : nullptr;
  Py_XDECREF(slice);
  return v;
}
PyObject* part_of(PyObject* batch, int name, PyObject* beg, PyObject* end) {
  PyObject* array = PyObject_GetAttr(batch, name_of[name]);
  PyObject* v = array ? part(array, beg, end) : nullptr;
  Py_XDECREF(array);
  return v;
}
// entries k and k + 1 of a list attribute of the batch (owned by the list, which the batch keeps)
bool range_of(PyObject* batch, int name, Py_ssize_t k, PyObject** beg, PyObject** end) {
  PyObject* list = PyObject_GetAttr(batch, name_of[name]);
  if (!list) return false;
  const bool ok = PyList_CheckExact(list) && k >= 0 && k + 1 < PyList_GET_SIZE(list);
  if (ok) {
    *beg = PyList_GET_ITEM(list, k);
    *end = PyList_GET_ITEM(list, k + 1);
  } else {
    PyErr_SetString(PyExc_IndexError, "system index out of range");
  }
  Py_DECREF(list);
  return ok;
}

PyObject* component_names;  // the tuple of component names, set by set_components

// The components of system k of the batch's energies (float64, systems x 15).
PyObject* components_of(PyObject* batch, Py_ssize_t k) {
  PyObject* array = PyObject_GetAttr(batch, name_of[N_ENERGY]);
  if (!array) return nullptr;
  Py_buffer view;
  const int rc = PyObject_GetBuffer(array, &view, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT);
  Py_DECREF(array);
  if (rc != 0) return nullptr;
  PyObject* out = nullptr;
  const Py_ssize_t n = component_names ? PyTuple_GET_SIZE(component_names) : 0;
  if (view.itemsize != 8 || k < 0 || 120 * (k + 1) > view.len || n != 14) {
    PyErr_SetString(PyExc_IndexError, "system index out of range");
  } else if ((out = PyDict_New()) != nullptr) {
    const double* e = static_cast<const double*>(view.buf) + 15 * k;
    for (Py_ssize_t c = 0; out && c < n; ++c) {
      PyObject* v = PyFloat_FromDouble(e[c]);
      if (!v || PyDict_SetItem(out, PyTuple_GET_ITEM(component_names, c), v) != 0) Py_CLEAR(out);
      Py_XDECREF(v);
    }
  }
  PyBuffer_Release(&view);
  return out;
}

// field(evaluation, name): reached for a field that is not set yet. An evaluation of a batch gets the field
// from the batch's arrays and keeps it.
PyObject* field(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "field takes an evaluation and a name");
    return nullptr;
  }
  PyObject *ev = args[0], *name = args[1], *value = nullptr;
  PyObject* dict = PyObject_GenericGetDict(ev, nullptr);
  if (!dict) return nullptr;
  PyObject* batch = PyDict_GetItemWithError(dict, name_of[N_BATCH]);  // borrowed
  PyObject* index = batch ? PyDict_GetItemWithError(dict, name_of[N_INDEX]) : nullptr;
  int which = N_FORCES;
  while (which <= N_COMPONENTS && name != name_of[which]) ++which;
  if (which > N_COMPONENTS && PyUnicode_Check(name)) {  // an equal name that is not the interned one
    which = N_FORCES;
    while (which <= N_COMPONENTS && PyUnicode_Compare(name, name_of[which]) != 0) ++which;
  }
  if (!batch || !index || which > N_COMPONENTS) {
    if (!PyErr_Occurred()) PyErr_SetObject(PyExc_AttributeError, name);
    Py_DECREF(dict);
    return nullptr;
  }
  Py_INCREF(batch);
  const Py_ssize_t k = PyLong_AsSsize_t(index);
  PyObject *beg = nullptr, *end = nullptr;
  if (k == -1 && PyErr_Occurred()) {
  } else if (which == N_COMPONENTS) {
    value = components_of(batch, k);
  } else if (which == N_DIPOLE) {
    PyObject* array = PyObject_GetAttr(batch, name_of[N_DIPOLE]);
    value = array ? PySequence_GetItem(array, k) : nullptr;
    Py_XDECREF(array);
  } else if (which == N_BONDS) {
    PyObject* all = PyObject_GetAttr(batch, name_of[N_BONDS]);
    if (all && PyTuple_CheckExact(all) && range_of(batch, N_CUT, k, &beg, &end)) {
      const Py_ssize_t n = PyTuple_GET_SIZE(all);
      value = PyTuple_New(n);
      for (Py_ssize_t q = 0; value && q < n; ++q) {
        PyObject* v = part(PyTuple_GET_ITEM(all, q), beg, end);
        if (v)
          PyTuple_SET_ITEM(value, q, v);
        else
          Py_CLEAR(value);
      }
    }
    Py_XDECREF(all);
  } else if (range_of(batch, N_OFFSETS, k, &beg, &end)) {
    value = part_of(batch, which, beg, end);
  }
  Py_DECREF(batch);
  if (value && PyDict_SetItem(dict, name, value) != 0) Py_CLEAR(value);
  if (!value && !PyErr_Occurred()) PyErr_SetObject(PyExc_AttributeError, name);
  Py_DECREF(dict);
  return value;
}

PyObject* set_components(PyObject*, PyObject* names) {
  if (!PyTuple_CheckExact(names)) {
    PyErr_SetString(PyExc_TypeError, "a tuple of names");
    return nullptr;
  }
  Py_XSETREF(component_names, Py_NewRef(names));
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"fill", fill, METH_VARARGS, "Pack a batch's symbols and positions; returns the requests left for Python."},
    {"guesses", guesses, METH_VARARGS,
     "Addresses of the requests' initial charges (0 for None); returns the requests left for Python."},
    {"items", items, METH_O, "The request tuples of keyword dicts, or None."},
    {"cells", cells, METH_VARARGS, "Fully periodic cells of a batch; returns those taken and those left for Python."},
    {"evaluations", evaluations, METH_VARARGS, "The result objects of a batch."},
    {"set_components", set_components, METH_O, "Names of the energy components."},
    {nullptr, nullptr, 0, nullptr},
};

PyMethodDef field_method = {"field", (PyCFunction)(void (*)(void))field, METH_FASTCALL,
                            "A field of an evaluation of a batch, made on first access."};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_xr_host", "Host-side batch packing.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

// `field` is an instance method: as a class attribute it binds the evaluation, like a Python function.
PyMODINIT_FUNC PyInit__xr_host(void) {
  for (int k = 0; k < N_NAMES; ++k)
    if (!name_of[k] && !(name_of[k] = PyUnicode_InternFromString(kNames[k]))) return nullptr;
  PyObject* m = PyModule_Create(&module);
  PyObject* f = m ? PyCFunction_New(&field_method, nullptr) : nullptr;
  PyObject* bound = f ? PyInstanceMethod_New(f) : nullptr;
  Py_XDECREF(f);
  if (!bound || PyModule_AddObjectRef(m, "field", bound) != 0) {
    Py_XDECREF(bound);
    Py_XDECREF(m);
    return nullptr;
  }
  Py_DECREF(bound);
  return m;
}
