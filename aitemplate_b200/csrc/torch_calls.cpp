// The host path of the eager calls (aitemplate_b200/kernels.py) and of Model.run_with_tensors: reads the tensors, allocates the
// output and calls the C entry point of libb200ait.so, in native code. A call of gemm_rcr at 256 x 3072 x 768 takes the GPU 6 us
// and took the host 12, of which the launch itself is 3 (here 6; a softmax 7 -> 4.3, seven row-wise calls 70 -> 28; run_with_tensors of an
// encoder layer at batch 1 70 -> 55 with the GPU's 45).
//
// Every function takes plain calls only (exact torch.Tensor or Parameter objects on the GPU, contiguous, shapes that fit) and
// returns None for anything else; the Python code behind it then runs as if this module were not there, and is the one
// place that refuses calls and says why. Nothing is kept from one call for the next.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <vector>

#include "b200ait.h"
#include "model_interface.h"

namespace {

// Addresses in the libb200ait.so that the package has loaded (bind()).
struct Library {
  decltype(&b200ait_gemm_rcr) gemm_rcr;
  decltype(&b200ait_gemm_rrr) gemm_rrr;
  decltype(&b200ait_gemm_rcr_scratch_bytes) scratch_bytes;
  decltype(&b200ait_mem_eff_attention) attention;
  decltype(&b200ait_flash_attention) flash_attention;
  decltype(&b200ait_layernorm) layernorm;
  decltype(&b200ait_softmax) softmax;
  decltype(&b200ait_concatenate) concatenate;
  decltype(&b200ait_split) split;
  decltype(&b200ait_permute) permute;
  decltype(&b200ait_last_error) last_error;
  decltype(&AITemplateModelContainerRun) run;
} lib;
PyTypeObject* parameter_type = nullptr;  // torch.nn.Parameter

// A tensor argument: null if the object is no plain tensor on the GPU, contiguous.
const at::Tensor* plain(PyObject* o) {
  if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass) && Py_TYPE(o) != parameter_type) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  // (a conjugated or negated view, a functorch wrapper or a fake tensor has no memory of its own to hand over)
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_conj() || t.is_neg()) return nullptr;
  if (t.unsafeGetTensorImpl()->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched,
                                                                     c10::DispatchKey::FuncTorchGradWrapper,
                                                                     c10::DispatchKey::Functionalize, c10::DispatchKey::Python})))
    return nullptr;
  return t.is_contiguous() ? &t : nullptr;
}
// an optional one: false if it is neither None nor plain
bool optional_plain(PyObject* o, const at::Tensor** t) {
  *t = o == Py_None ? nullptr : plain(o);
  return o == Py_None || *t != nullptr;
}
void* pointer(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
int dtype_code(const at::Tensor& t) {
  return t.scalar_type() == at::kHalf ? static_cast<int>(AITemplateDtype::kHalf)
                                      : t.scalar_type() == at::kBFloat16 ? static_cast<int>(AITemplateDtype::kBFloat16) : 0;
}
b200ait_stream_t current_stream() { return reinterpret_cast<b200ait_stream_t>(c10::cuda::getCurrentCUDAStream().stream()); }

PyObject* unhandled() { Py_RETURN_NONE; }
PyObject* failed(const char* name) {
  return PyErr_Format(PyExc_RuntimeError, "Error in function: %s: %s", name, lib.last_error());
}
// A C++ exception (out of memory, above all) sends the call to the Python code, which meets the same one and raises it as torch does.
template <class F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const std::exception&) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}
// the entry point itself, without the interpreter's lock
template <class F>
int unlocked(F&& f) {
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = f();
  Py_END_ALLOW_THREADS;
  return code;
}
bool as_int(PyObject* o, int64_t* v) {
  if (!PyLong_Check(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool as_double(PyObject* o, double* v) {
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
  *v = PyFloat_AsDouble(o);
  if (*v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool as_dim(PyObject* o, int64_t rank, int64_t* v) {  // Python's dim % rank
  if (rank == 0 || !as_int(o, v)) return false;
  *v = ((*v % rank) + rank) % rank;
  return true;
}

// gemm_rcr(x, w, bias, d0, d1, epilogue code, alpha, tile_n, split_k)
PyObject* gemm_rcr(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 9) return unhandled();
    const at::Tensor *x = plain(args[0]), *w = plain(args[1]), *bias, *d0, *d1;
    int64_t epilogue, tile_n, split_k, ws = 0;
    double alpha;
    if (!x || !w || !optional_plain(args[2], &bias) || !optional_plain(args[3], &d0) || !optional_plain(args[4], &d1) ||
        !as_int(args[5], &epilogue) || !as_double(args[6], &alpha) || !as_int(args[7], &tile_n) || !as_int(args[8], &split_k))
      return unhandled();
    if (x->dim() < 1 || w->dim() != 2 || dtype_code(*x) == 0) return unhandled();
    const int64_t k = x->size(-1), n = w->size(0);
    if (k == 0 || w->size(1) != k || x->numel() == 0 || n == 0) return unhandled();
    const int64_t m = x->numel() / k;
    // (a launch that takes scratch goes the long way)
    if (split_k != 1 && (lib.scratch_bytes(m, n, k, static_cast<int>(tile_n), static_cast<int>(split_k), &ws) != 0 || ws != 0))
      return unhandled();
    std::vector<int64_t> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = n;
    at::Tensor out = x->new_empty(shape);
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] {
          return lib.gemm_rcr(pointer(x), pointer(w), pointer(bias), pointer(d0), pointer(d1), out.data_ptr(), 1, m, n, k, k, k, n, n,
                              0, 0, 0, 0, static_cast<int>(epilogue), dtype_code(*x), static_cast<float>(alpha), 0, 1, 1, 1,
                              static_cast<int>(tile_n), nullptr, 0, static_cast<int>(split_k), stream);
        }))
      return failed("b200ait_gemm_rcr");
    return THPVariable_Wrap(std::move(out));
  });
}

// bmm(a, b, alpha, tile_n, b is stored [K, N])
PyObject* bmm(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 5) return unhandled();
    const at::Tensor *a = plain(args[0]), *b = plain(args[1]);
    int64_t tile_n;
    double alpha;
    if (!a || !b || !as_double(args[2], &alpha) || !as_int(args[3], &tile_n)) return unhandled();
    const bool row_major = args[4] == Py_True;
    const int64_t da = a->dim(), db = b->dim();
    if (da < 2 || da > 3 || db < 2 || db > 3 || dtype_code(*a) == 0) return unhandled();
    const int64_t ba = da == 3 ? a->size(0) : 1, bb = db == 3 ? b->size(0) : 1;
    const int64_t m = a->size(da - 2), k = a->size(da - 1);
    const int64_t n = b->size(row_major ? db - 1 : db - 2), k2 = b->size(row_major ? db - 2 : db - 1);
    if (k != k2 || !(ba == bb || ba == 1 || bb == 1) || a->numel() == 0 || b->numel() == 0) return unhandled();
    const int64_t batch = std::max(ba, bb), a_bs = ba == 1 && batch > 1 ? 0 : m * k, b_bs = bb == 1 && batch > 1 ? 0 : n * k;
    at::Tensor out = a->new_empty({batch, m, n});
    const b200ait_stream_t stream = current_stream();
    const int code = unlocked([&] {
      return row_major ? lib.gemm_rrr(pointer(a), pointer(b), nullptr, nullptr, nullptr, out.data_ptr(), batch, m, n, k, k, n, n, n, a_bs,
                                      b_bs, m * n, m * n, 0, dtype_code(*a), static_cast<float>(alpha), static_cast<int>(tile_n),
                                      nullptr, 0, 1, stream)
                       : lib.gemm_rcr(pointer(a), pointer(b), nullptr, nullptr, nullptr, out.data_ptr(), batch, m, n, k, k, k, n, n, a_bs,
                                      b_bs, m * n, m * n, 0, dtype_code(*a), static_cast<float>(alpha), 0, 1, 1, 1,
                                      static_cast<int>(tile_n), nullptr, 0, 1, stream);
    });
    if (code) return failed(row_major ? "b200ait_gemm_rrr" : "b200ait_gemm_rcr");
    return THPVariable_Wrap(std::move(out));
  });
}

// the softmax scale: a number, or None for 1 / sqrt(d)
bool as_scale(PyObject* o, int64_t d, double* v) {
  if (o != Py_None) return as_double(o, v);
  *v = d != 0 ? 1.0 / std::sqrt(static_cast<double>(d)) : 1.0;
  return true;
}

// mem_eff_attention(q, k, v, causal, scale, lengths_kv, lengths_q)
PyObject* mem_eff_attention(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 7) return unhandled();
    const at::Tensor *q = plain(args[0]), *k = plain(args[1]), *v = plain(args[2]), *lengths[2];
    if (!q || !k || !v || !optional_plain(args[5], &lengths[0]) || !optional_plain(args[6], &lengths[1])) return unhandled();
    if (q->dim() != 4 || k->dim() != 4 || v->dim() != 4 || dtype_code(*q) == 0 || !PyBool_Check(args[3])) return unhandled();
    const int64_t b = q->size(0), h = q->size(1), sq = q->size(2), d = q->size(3), skv = k->size(2), dv = v->size(3);
    double scale;
    if (!as_scale(args[4], d, &scale) || q->numel() == 0 || k->numel() == 0 || v->numel() == 0) return unhandled();
    for (const at::Tensor* t : lengths)
      if (t != nullptr && (t->scalar_type() != at::kInt || t->numel() != b)) return unhandled();
    at::Tensor out = q->new_empty({b, sq, h, dv});
    const b200ait_stream_t stream = current_stream();
    const int causal = args[3] == Py_True;
    if (unlocked([&] {
          return lib.attention(out.data_ptr(), pointer(q), pointer(k), pointer(v), b, skv, sq, static_cast<int>(h),
                               static_cast<int>(d), static_cast<int>(dv), static_cast<float>(scale), causal,
                               static_cast<const int32_t*>(pointer(lengths[0])), static_cast<const int32_t*>(pointer(lengths[1])),
                               dtype_code(*q), stream);
        }))
      return failed("b200ait_mem_eff_attention");
    return THPVariable_Wrap(std::move(out));
  });
}

// flash_attention(qkv, cu_seqlens, max_seq_len, causal, scale)
PyObject* flash_attention(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 5) return unhandled();
    const at::Tensor *qkv = plain(args[0]), *cu = plain(args[1]);
    int64_t bound;
    double scale;
    if (!qkv || !cu || qkv->dim() != 4 || qkv->size(1) != 3 || cu->scalar_type() != at::kInt || dtype_code(*qkv) == 0 ||
        !as_int(args[2], &bound) || bound != static_cast<int>(bound) || !PyBool_Check(args[3]) || qkv->numel() == 0)
      return unhandled();
    const int64_t total = qkv->size(0), h = qkv->size(2), d = qkv->size(3);
    if (!as_scale(args[4], d, &scale)) return unhandled();
    at::Tensor out = qkv->new_empty({total, h, d});
    const b200ait_stream_t stream = current_stream();
    const int causal = args[3] == Py_True;
    if (unlocked([&] {
          return lib.flash_attention(out.data_ptr(), pointer(qkv), static_cast<const int*>(pointer(cu)), nullptr, nullptr,
                                     static_cast<int>(cu->numel() - 1), static_cast<int>(bound), static_cast<int>(h),
                                     static_cast<int>(d), 0.f, static_cast<float>(scale), causal, 0, total, dtype_code(*qkv), stream);
        }))
      return failed("b200ait_flash_attention");
    return THPVariable_Wrap(std::move(out));
  });
}

// layernorm(x, gamma, beta, eps, normalized_ndim)
PyObject* layernorm(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 5) return unhandled();
    const at::Tensor *x = plain(args[0]), *gamma, *beta;
    int64_t dims;
    double eps;
    if (!x || !optional_plain(args[1], &gamma) || !optional_plain(args[2], &beta) || !as_double(args[3], &eps) ||
        !as_int(args[4], &dims) || dims < 0 || dims > x->dim() || x->numel() == 0 || dtype_code(*x) == 0)
      return unhandled();
    int64_t n = 1;
    for (int64_t i = x->dim() - dims; i < x->dim(); ++i) n *= x->size(i);
    at::Tensor out = at::empty_like(*x);
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] {
          return lib.layernorm(out.data_ptr(), pointer(x), pointer(gamma), pointer(beta), x->numel() / n, n, static_cast<float>(eps),
                               0, 0, dtype_code(*x), stream);
        }))
      return failed("b200ait_layernorm");
    return THPVariable_Wrap(std::move(out));
  });
}

// softmax(x, dim)
PyObject* softmax(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 2) return unhandled();
    const at::Tensor* x = plain(args[0]);
    int64_t dim;
    if (!x || x->numel() == 0 || dtype_code(*x) == 0 || !as_dim(args[1], x->dim(), &dim)) return unhandled();
    int64_t outer = 1, inner = 1;
    for (int64_t i = 0; i < x->dim(); ++i) (i < dim ? outer : inner) *= i == dim ? 1 : x->size(i);
    at::Tensor out = at::empty_like(*x);
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] { return lib.softmax(pointer(x), out.data_ptr(), outer, x->size(dim), inner, dtype_code(*x), stream); }))
      return failed("b200ait_softmax");
    return THPVariable_Wrap(std::move(out));
  });
}

// concatenate(tensors, dim)
PyObject* concatenate(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 2 || (!PyList_Check(args[0]) && !PyTuple_Check(args[0]))) return unhandled();
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(args[0]);
    if (n == 0) return unhandled();
    std::vector<const void*> pointers;
    std::vector<const int64_t*> shapes;
    // The list may change while the lock is released, or under a dispatch mode while the output is allocated: from here on the
    // tensors are read through `held` alone.
    std::vector<at::Tensor> held;
    std::vector<int64_t> shape;
    int64_t dim = 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
      const at::Tensor* t = plain(PySequence_Fast_GET_ITEM(args[0], i));
      if (!t || t->numel() == 0) return unhandled();
      if (i == 0) {
        shape.assign(t->sizes().begin(), t->sizes().end());
        if (!as_dim(args[1], t->dim(), &dim)) return unhandled();
      } else {
        if (t->dim() != held[0].dim() || t->scalar_type() != held[0].scalar_type()) return unhandled();
        for (int64_t j = 0; j < t->dim(); ++j)
          if (j != dim && t->size(j) != shape[j]) return unhandled();
        shape[dim] += t->size(dim);
      }
      pointers.push_back(t->data_ptr());
      shapes.push_back(t->sizes().data());
      held.push_back(*t);
    }
    const std::vector<uint8_t> masks(n, 1);
    std::vector<int64_t> out_shape(shape.size());
    at::Tensor out = held[0].new_empty(shape);
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] {
          return lib.concatenate(out.data_ptr(), out_shape.data(), pointers.data(), shapes.data(), masks.data(), dim, held[0].dim(), n,
                                 static_cast<int64_t>(held[0].element_size()), stream);
        }))
      return failed("b200ait_concatenate");
    return THPVariable_Wrap(std::move(out));
  });
}

// split(x, size, dim): blocks of `size`, the last one shorter
PyObject* split(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 3) return unhandled();
    const at::Tensor* x = plain(args[0]);
    int64_t size, dim;
    if (!x || x->numel() == 0 || PyBool_Check(args[1]) || !as_int(args[1], &size) || size <= 0 || !as_dim(args[2], x->dim(), &dim))
      return unhandled();
    std::vector<int64_t> sizes, shape(x->sizes().begin(), x->sizes().end());
    for (int64_t at = 0; at < x->size(dim); at += size) sizes.push_back(std::min(size, x->size(dim) - at));
    std::vector<at::Tensor> outs;
    std::vector<void*> pointers;
    for (const int64_t s : sizes) {
      shape[dim] = s;
      outs.push_back(x->new_empty(shape));
      pointers.push_back(outs.back().data_ptr());
    }
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] {
          return lib.split(pointers.data(), nullptr, pointer(x), x->sizes().data(), static_cast<int64_t>(sizes.size()), sizes.data(), dim,
                           x->dim(), static_cast<int64_t>(x->element_size()), stream);
        }))
      return failed("b200ait_split");
    PyObject* list = PyList_New(static_cast<Py_ssize_t>(outs.size()));
    if (!list) return nullptr;
    for (size_t i = 0; i < outs.size(); ++i) PyList_SET_ITEM(list, static_cast<Py_ssize_t>(i), THPVariable_Wrap(std::move(outs[i])));
    return list;
  });
}

// permute(x, dims)
PyObject* permute(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 2 || (!PyList_Check(args[1]) && !PyTuple_Check(args[1]))) return unhandled();
    const at::Tensor* x = plain(args[0]);
    if (!x || x->numel() == 0 || PySequence_Fast_GET_SIZE(args[1]) != x->dim()) return unhandled();
    std::vector<int64_t> dims, shape;
    std::vector<bool> seen(static_cast<size_t>(x->dim()), false);
    for (int64_t i = 0; i < x->dim(); ++i) {
      int64_t d;
      if (!as_dim(PySequence_Fast_GET_ITEM(args[1], i), x->dim(), &d) || seen[d]) return unhandled();
      seen[d] = true;
      dims.push_back(d), shape.push_back(x->size(d));
    }
    at::Tensor out = x->new_empty(shape);
    const b200ait_stream_t stream = current_stream();
    if (unlocked([&] {
          return lib.permute(pointer(x), out.data_ptr(), x->sizes().data(), dims.data(), x->dim(),
                             static_cast<int64_t>(x->element_size()), stream);
        }))
      return failed("b200ait_permute");
    return THPVariable_Wrap(std::move(out));
  });
}

// One side (inputs or outputs) of a run, in the order of the model's indexes.
struct Side {
  std::vector<AITData> data;
  std::vector<const at::Tensor*> tensors;
  std::vector<PyObject*> names;
  std::vector<size_t> given_order;  // the indexes in the order of the caller's dictionary
  bool read(PyObject* given, PyObject* index_of) {
    if (!PyDict_CheckExact(given) || !PyDict_CheckExact(index_of) || PyDict_GET_SIZE(given) != PyDict_GET_SIZE(index_of)) return false;
    const size_t n = static_cast<size_t>(PyDict_GET_SIZE(given));
    data.resize(n), tensors.assign(n, nullptr), names.assign(n, nullptr);
    PyObject *name, *value;
    for (Py_ssize_t at = 0; PyDict_Next(given, &at, &name, &value);) {
      PyObject* index = PyDict_GetItemWithError(index_of, name);
      int64_t i;
      if (!index || !as_int(index, &i) || i < 0 || i >= static_cast<int64_t>(n) || names[i]) {
        PyErr_Clear();
        return false;
      }
      const at::Tensor* t = plain(value);
      if (!t) return false;
      AITemplateDtype dtype;
      switch (t->scalar_type()) {
        case at::kHalf: dtype = AITemplateDtype::kHalf; break;
        case at::kBFloat16: dtype = AITemplateDtype::kBFloat16; break;
        case at::kFloat: dtype = AITemplateDtype::kFloat; break;
        case at::kInt: dtype = AITemplateDtype::kInt; break;
        case at::kLong: dtype = AITemplateDtype::kLong; break;
        case at::kBool: dtype = AITemplateDtype::kBool; break;
        default: return false;
      }
      names[i] = name, tensors[i] = t, given_order.push_back(static_cast<size_t>(i));
      data[i] = AITData(t->data_ptr(), AITemplateParamShape(t->sizes().data(), static_cast<size_t>(t->dim())), dtype);
    }
    return true;
  }
};

// run_model(handle, inputs, outputs, input name -> index, output name -> index, dimensions of each output, stream or None, sync,
// graph mode) -> {name: the output as the run shaped it}, in the order of `outputs`
PyObject* run_model(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 9) return unhandled();
    int64_t handle, stream = 0;
    Side in, out;
    if (!as_int(args[0], &handle) || handle == 0 || !in.read(args[1], args[3]) || !out.read(args[2], args[4]) ||
        !PyList_CheckExact(args[5]) || PyList_GET_SIZE(args[5]) != static_cast<Py_ssize_t>(out.data.size()) ||
        !PyBool_Check(args[7]) || !PyBool_Check(args[8]))
      return unhandled();
    if (args[6] == Py_None)
      stream = reinterpret_cast<int64_t>(current_stream());
    else if (!as_int(args[6], &stream))
      return unhandled();
    std::vector<std::vector<int64_t>> shapes(out.data.size());
    std::vector<int64_t*> shape_pointers;
    for (size_t i = 0; i < shapes.size(); ++i) {
      int64_t dims;
      if (!as_int(PyList_GET_ITEM(args[5], static_cast<Py_ssize_t>(i)), &dims) || dims != out.tensors[i]->dim()) return unhandled();
      shapes[i].resize(static_cast<size_t>(dims));
      shape_pointers.push_back(shapes[i].data());
    }
    const bool sync = args[7] == Py_True, graph_mode = args[8] == Py_True;
    // The dictionaries may change while the lock is released: what the run reads is held.
    std::vector<at::Tensor> held;
    for (const Side* side : {&in, &out})
      for (const at::Tensor* t : side->tensors) held.push_back(*t);
    std::vector<PyObject*> names = out.names;
    for (PyObject* name : names) Py_INCREF(name);
    const int code = unlocked([&] {
      return static_cast<int>(lib.run(reinterpret_cast<AITemplateModelHandle>(handle), in.data.data(), in.data.size(), out.data.data(),
                                      out.data.size(), reinterpret_cast<AITemplateStreamHandle>(stream), sync, graph_mode,
                                      shape_pointers.data()));
    });
    PyObject* result = code ? failed("AITemplateModelContainerRun") : PyDict_New();
    for (const size_t i : out.given_order) {
      if (result && !code) {
        const at::Tensor& t = held[in.tensors.size() + i];
        int64_t numel = 1;
        for (const int64_t s : shapes[i]) numel *= s;
        PyObject* view = nullptr;
        try {
          view = THPVariable_Wrap(numel == t.numel() ? t.view(shapes[i]) : t.flatten().narrow(0, 0, numel).reshape(shapes[i]));
        } catch (const std::exception& e) {
          PyErr_SetString(PyExc_RuntimeError, e.what());
        }
        if (!view || PyDict_SetItem(result, names[i], view) != 0) Py_CLEAR(result);
        Py_XDECREF(view);
      }
      Py_DECREF(names[i]);
    }
    return result;
  });
}

// bind(addresses of the library's entry points in the order of Library, torch.nn.Parameter)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  constexpr Py_ssize_t kEntries = sizeof(Library) / sizeof(void*);
  if (n_args != 2 || !PyTuple_Check(args[0]) || PyTuple_GET_SIZE(args[0]) != kEntries || !PyType_Check(args[1]))
    return PyErr_Format(PyExc_TypeError, "bind: expected %zd addresses and a type", kEntries);
  void* at[kEntries];
  for (Py_ssize_t i = 0; i < kEntries; ++i) {
    at[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(args[0], i));
    if (PyErr_Occurred()) return nullptr;
  }
  static_assert(sizeof(at) == sizeof(lib), "one address per entry");
  memcpy(&lib, at, sizeof(lib));
  parameter_type = reinterpret_cast<PyTypeObject*>(args[1]);
  Py_INCREF(args[1]);
  Py_RETURN_NONE;
}

#define B200AIT_METHOD(NAME) {#NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&NAME)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B200AIT_METHOD(bind),
                         B200AIT_METHOD(gemm_rcr),
                         B200AIT_METHOD(bmm),
                         B200AIT_METHOD(mem_eff_attention),
                         B200AIT_METHOD(flash_attention),
                         B200AIT_METHOD(layernorm),
                         B200AIT_METHOD(softmax),
                         B200AIT_METHOD(concatenate),
                         B200AIT_METHOD(split),
                         B200AIT_METHOD(permute),
                         B200AIT_METHOD(run_model),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_torch_calls() { return PyModule_Create(&module); }
