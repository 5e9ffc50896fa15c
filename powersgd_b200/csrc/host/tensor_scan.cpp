// Checks and address keys of whole lists of tensors, as a CPython extension against PyTorch's C++ interface.
//
// An eager step asks every parameter, gradient and momentum buffer for its type, layout and address. At
// 0.1 to 0.5 us per question in Python that was most of a step of ResNet-18 (62 parameters): 190 us of
// host time beside 113 us of kernels. Here a question takes some 10 ns. Nothing is remembered from one
// call for the next. A function answers None for objects it does not know (subclasses of Tensor, tensors
// of a transform, lists that are something else); the caller then asks in Python (ops/scan.py).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/TensorSubclassLikeUtils.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <exception>
#include <vector>

namespace {

// The tensor behind `object` when it is a plain one (exactly torch.Tensor or torch.nn.Parameter, strided, with
// memory of its own), else null.
const at::Tensor* plain(PyObject* object) {
  if (!THPVariable_CheckExact(object)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(object);
  if (!t.defined() || t.layout() != at::kStrided || !t.unsafeGetTensorImpl()->has_storage() || at::isTensorSubclassLike(t)) return nullptr;
  return &t;
}

// utils.is_dense
bool dense(const at::Tensor& t) { return t.is_contiguous() || (t.dim() == 4 && t.is_contiguous(at::MemoryFormat::ChannelsLast)); }

// utils.same_layout
bool same_layout(const at::Tensor& a, const at::Tensor& b) {
  if (a.sizes() != b.sizes()) return false;
  const auto n = a.sizes(), sa = a.strides(), sb = b.strides();
  for (size_t i = 0; i < n.size(); ++i)
    if (n[i] != 1 && sa[i] != sb[i]) return false;
  return true;
}

struct Sequence {   // a list or tuple, borrowed items
  PyObject* fast;
  explicit Sequence(PyObject* object) : fast(PyList_Check(object) || PyTuple_Check(object) ? PySequence_Fast(object, "") : nullptr) {}
  ~Sequence() { Py_XDECREF(fast); }
  Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(fast); }
  PyObject* operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(fast, i); }
};

PyObject* bytes_of(const std::vector<uint64_t>& words) {
  return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(words.data()), (Py_ssize_t)(words.size() * sizeof(uint64_t)));
}

template <class F>
PyObject* guarded(F body) {   // no C++ exception leaves the module
  try {
    return body();
  } catch (const std::exception& e) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// addresses(tensors): the addresses of a list as bytes, 0 for None.
PyObject* addresses(PyObject*, PyObject* list) {
  return guarded([&]() -> PyObject* {
    Sequence items(list);
    if (!items.fast) Py_RETURN_NONE;
    std::vector<uint64_t> words;
    words.reserve(items.size());
    for (Py_ssize_t i = 0; i < items.size(); ++i) {
      if (items[i] == Py_None) {
        words.push_back(0);
        continue;
      }
      const at::Tensor* t = plain(items[i]);
      if (t == nullptr) Py_RETURN_NONE;
      words.push_back((uint64_t)t->data_ptr());
    }
    return bytes_of(words);
  });
}

// grad_addresses(parameters): the addresses of their gradients as bytes; None where one has none.
PyObject* grad_addresses(PyObject*, PyObject* list) {
  return guarded([&]() -> PyObject* {
    Sequence items(list);
    if (!items.fast) Py_RETURN_NONE;
    std::vector<uint64_t> words;
    words.reserve(items.size());
    for (Py_ssize_t i = 0; i < items.size(); ++i) {
      const at::Tensor* t = plain(items[i]);
      if (t == nullptr || !t->grad().defined()) Py_RETURN_NONE;
      const at::Tensor& g = t->grad();
      if (g.layout() != at::kStrided || !g.unsafeGetTensorImpl()->has_storage() || at::isTensorSubclassLike(g)) Py_RETURN_NONE;
      words.push_back((uint64_t)g.data_ptr());
    }
    return bytes_of(words);
  });
}

// usable(tensors, contiguous): are all of them float32 tensors on a GPU, dense (contiguous != 0: contiguous)?
PyObject* usable(PyObject*, PyObject* args) {
  return guarded([&]() -> PyObject* {
    PyObject* list;
    int contiguous;
    if (!PyArg_ParseTuple(args, "Op", &list, &contiguous)) return nullptr;
    Sequence items(list);
    if (!items.fast) Py_RETURN_NONE;
    for (Py_ssize_t i = 0; i < items.size(); ++i) {
      const at::Tensor* t = plain(items[i]);
      if (t == nullptr) Py_RETURN_NONE;
      if (!t->is_cuda() || t->scalar_type() != at::kFloat || !(contiguous ? t->is_contiguous() : dense(*t))) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
  });
}

// sizes(tensors): the numbers of elements as bytes.
PyObject* sizes(PyObject*, PyObject* list) {
  return guarded([&]() -> PyObject* {
    Sequence items(list);
    if (!items.fast) Py_RETURN_NONE;
    std::vector<uint64_t> words;
    words.reserve(items.size());
    for (Py_ssize_t i = 0; i < items.size(); ++i) {
      const at::Tensor* t = plain(items[i]);
      if (t == nullptr) Py_RETURN_NONE;
      words.push_back((uint64_t)t->numel());
    }
    return bytes_of(words);
  });
}

// step_fits(param_groups, state): what the fused optimizer step needs of every group, parameter, gradient and
// momentum buffer (PowerSGD.supports_fused_step).
PyObject* step_fits(PyObject*, PyObject* args) {
  return guarded([&]() -> PyObject* {
    PyObject *group_list, *state;
    if (!PyArg_ParseTuple(args, "OO", &group_list, &state)) return nullptr;
    Sequence groups(group_list);
    if (!groups.fast || !PyDict_Check(state)) Py_RETURN_NONE;
    for (Py_ssize_t g = 0; g < groups.size(); ++g) {
      PyObject* group = groups[g];
      if (!PyDict_Check(group)) Py_RETURN_NONE;
      for (const char* flag : {"maximize", "differentiable"}) {
        PyObject* value = PyDict_GetItemString(group, flag);
        if (value == nullptr || value == Py_False) continue;
        if (value != Py_True) Py_RETURN_NONE;
        Py_RETURN_FALSE;
      }
      PyObject* list = PyDict_GetItemString(group, "params");
      if (list == nullptr) Py_RETURN_NONE;
      Sequence params(list);
      if (!params.fast) Py_RETURN_NONE;
      Py_ssize_t buffers = 0;
      for (Py_ssize_t i = 0; i < params.size(); ++i) {
        const at::Tensor* p = plain(params[i]);
        if (p == nullptr) Py_RETURN_NONE;
        const at::Tensor& grad = p->grad();
        if (!grad.defined() || p->scalar_type() != at::kFloat || !dense(*p)) Py_RETURN_FALSE;
        if (grad.layout() != at::kStrided || at::isTensorSubclassLike(grad)) Py_RETURN_NONE;
        if (!same_layout(grad, *p)) Py_RETURN_FALSE;
        PyObject* own = PyDict_GetItemWithError(state, params[i]);
        if (own == nullptr) {
          if (PyErr_Occurred()) {
            PyErr_Clear();
            Py_RETURN_NONE;
          }
          continue;
        }
        if (!PyDict_Check(own)) Py_RETURN_NONE;
        PyObject* buffer = PyDict_GetItemString(own, "momentum_buffer");
        if (buffer == nullptr || buffer == Py_None) continue;
        const at::Tensor* m = plain(buffer);
        if (m == nullptr) Py_RETURN_NONE;
        ++buffers;
        if (!same_layout(*m, *p)) Py_RETURN_FALSE;
      }
      if (buffers != 0 && buffers != params.size()) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
  });
}

PyMethodDef methods[] = {
    {"addresses", addresses, METH_O, nullptr},     {"grad_addresses", grad_addresses, METH_O, nullptr}, {"usable", usable, METH_VARARGS, nullptr},
    {"sizes", sizes, METH_O, nullptr},             {"step_fits", step_fits, METH_VARARGS, nullptr},     {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tensor_scan", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tensor_scan() {
  PyObject* m = PyModule_Create(&module);
  // what this was compiled for, which the loader compares (csrc/build.py, scan_target)
  if (m != nullptr && PyModule_AddStringConstant(m, "target", PSGD_SCAN_TARGET) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
