// b2_native.cpp — CPython extension between the package's Column / Table / GroupBy objects and the C ABI of
// include/b2_groupby.h: reads the column objects into b2_column_view structs, hands the library torch's caching
// allocator, and turns the owning result columns into Column objects.
//
// Why it is native: a call on a thousand rows spends its time on the host.  With the structs built field by field
// through ctypes and every result buffer allocated by a Python callback, 70 of such a call's 112 us were Python
// (create 9, requests 13, allocation callbacks ~20, adopting the results 23, releasing 4).
//
// The GIL is released while the library runs; the allocator callbacks need none.
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/autograd/python_variable.h>
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <deque>
#include <vector>

#include "../../include/b2_groupby.h"

namespace {

// ------------------------------------------------------------------------------ names and classes
PyObject *n_type_id, *n_scale, *n_size, *n_null_count, *n_data, *n_mask, *n_offset, *n_offsets, *n_offsets_type, *n_children,
  *n_values, *n_aggregations, *n_kind, *n_ddof;
PyObject *cls_table = nullptr, *fn_adopt = nullptr, *fn_check = nullptr;
PyObject* type_ids[B2_STRUCT + 1] = {};  // TypeId members by value

int width_of(int t)
{
  switch (t) {
    case B2_INT8: case B2_UINT8: case B2_BOOL8: return 1;
    case B2_INT16: case B2_UINT16: return 2;
    case B2_INT32: case B2_UINT32: case B2_FLOAT32: case B2_TIMESTAMP_DAYS: case B2_DURATION_DAYS: case B2_DECIMAL32: return 4;
    case B2_DECIMAL128: return 16;
    case B2_EMPTY: case B2_DICTIONARY32: case B2_STRING: case B2_LIST: case B2_STRUCT: return 0;
    default: return 8;
  }
}

struct Ref {  // owned reference
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};
struct PyFailed {};  // a Python exception is set

long long int_attr(PyObject* o, PyObject* name)
{
  Ref v(PyObject_GetAttr(o, name));
  if (!v.p) throw PyFailed{};
  const long long x = PyLong_AsLongLong(v.p);
  if (x == -1 && PyErr_Occurred()) throw PyFailed{};
  return x;
}

// device pointer and element count of a tensor attribute (None: nullptr, 0); notes the device of the first CUDA tensor
void* tensor_attr(PyObject* o, PyObject* name, int64_t* numel, int* device)
{
  Ref v(PyObject_GetAttr(o, name));
  if (!v.p) throw PyFailed{};
  if (numel) *numel = 0;
  if (v.p == Py_None) return nullptr;
  if (!THPVariable_Check(v.p)) {
    PyErr_SetString(PyExc_TypeError, "a column's buffers are torch tensors");
    throw PyFailed{};
  }
  const at::Tensor& t = THPVariable_Unpack(v.p);
  if (numel) *numel = t.numel();
  if (device && *device < 0 && t.is_cuda()) *device = t.get_device();
  return t.data_ptr();
}

// ------------------------------------------------------------------------------ views
using Kids = std::deque<std::vector<b2_column_view>>;

b2_column_view view_of(PyObject* col, Kids& kids, int* device)
{
  b2_column_view v{};
  int64_t numel = 0;
  v.type_id = (int32_t)int_attr(col, n_type_id);
  v.scale = (int32_t)int_attr(col, n_scale);
  v.size = (int32_t)int_attr(col, n_size);
  v.offset = (int32_t)int_attr(col, n_offset);
  void* data = tensor_attr(col, n_data, &numel, device);
  v.data = numel ? data : nullptr;
  v.null_mask = (const uint32_t*)tensor_attr(col, n_mask, nullptr, device);
  v.null_count = v.null_mask ? (int32_t)int_attr(col, n_null_count) : 0;
  if (v.type_id == B2_STRING) {
    b2_column_view o{};
    o.type_id = (int32_t)int_attr(col, n_offsets_type);
    o.size = v.size + 1;
    void* p = tensor_attr(col, n_offsets, &numel, device);
    o.data = numel ? p : nullptr;
    kids.emplace_back(1, o);
  } else if (v.type_id == B2_DICTIONARY32 || v.type_id == B2_STRUCT) {
    Ref list(PyObject_GetAttr(col, n_children));
    if (!list.p) throw PyFailed{};
    if (list.p == Py_None) return v;
    Ref fast(PySequence_Fast(list.p, "children is not a sequence"));
    if (!fast.p) throw PyFailed{};
    std::vector<b2_column_view> ks;
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(fast.p); ++i)
      ks.push_back(view_of(PySequence_Fast_GET_ITEM(fast.p, i), kids, device));
    if (ks.empty()) return v;
    kids.push_back(std::move(ks));
  } else {
    return v;
  }
  v.num_children = (int32_t)kids.back().size();
  v.children = kids.back().data();
  return v;
}

struct Requests {
  std::vector<b2_aggregation_request> reqs;
  std::deque<std::vector<b2_aggregation>> aggs;
};
void read_requests(PyObject* list, Requests& r, Kids& kids, int* device)
{
  Ref fast(PySequence_Fast(list, "requests is not a sequence"));
  if (!fast.p) throw PyFailed{};
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast.p);
  r.reqs.reserve((size_t)n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* q = PySequence_Fast_GET_ITEM(fast.p, i);
    Ref values(PyObject_GetAttr(q, n_values)), list_(PyObject_GetAttr(q, n_aggregations));
    if (!values.p || !list_.p) throw PyFailed{};
    Ref as(PySequence_Fast(list_.p, "aggregations is not a sequence"));
    if (!as.p) throw PyFailed{};
    const Py_ssize_t na = PySequence_Fast_GET_SIZE(as.p);
    r.aggs.emplace_back((size_t)na);
    for (Py_ssize_t a = 0; a < na; ++a) {
      PyObject* agg = PySequence_Fast_GET_ITEM(as.p, a);
      r.aggs.back()[(size_t)a] = b2_aggregation{(int32_t)int_attr(agg, n_kind), (int32_t)int_attr(agg, n_ddof)};
    }
    b2_aggregation_request c{};
    c.values = view_of(values.p, kids, device);
    c.num_aggregations = (int32_t)na;
    c.aggregations = r.aggs.back().data();
    r.reqs.push_back(c);
  }
}

// ------------------------------------------------------------------------------ result buffers
struct Buffers {  // the buffers the library asked for during one call
  struct Item { void* p; size_t bytes; c10::DataPtr own; };
  std::vector<Item> live;
};
void* take_buffer(size_t bytes, void*, void* ctx)
{
  try {
    if (bytes < 8) bytes = 8;
    c10::DataPtr d = c10::cuda::CUDACachingAllocator::get()->allocate(bytes);
    void* p = d.get();
    ((Buffers*)ctx)->live.push_back(Buffers::Item{p, bytes, std::move(d)});
    return p;
  } catch (...) {
    return nullptr;
  }
}
void give_buffer(void* p, size_t, void*, void* ctx)
{
  auto& live = ((Buffers*)ctx)->live;
  for (size_t i = 0; i < live.size(); ++i)
    if (live[i].p == p) { live[i] = std::move(live.back()); live.pop_back(); return; }
}

// the buffer as a uint8 tensor of at most `used` bytes (0: all of it): a call that allocated its result before it knew
// the group count hands over buffers larger than the column
PyObject* as_tensor(Buffers& b, void*& p, size_t used)
{
  if (!p) Py_RETURN_NONE;
  for (auto& it : b.live) {
    if (it.p != p) continue;
    p = nullptr;
    const size_t n = used && used < it.bytes ? used : it.bytes;
    c10::Storage st(c10::Storage::use_byte_size_t(), it.bytes, std::move(it.own), c10::cuda::CUDACachingAllocator::get(), false);
    at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(std::move(st), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                            caffe2::TypeMeta::Make<uint8_t>());
    t.unsafeGetTensorImpl()->set_sizes_contiguous({(int64_t)n});
    if (&it != &b.live.back()) it = std::move(b.live.back());
    b.live.pop_back();
    return THPVariable_Wrap(std::move(t));
  }
  PyErr_SetString(PyExc_RuntimeError, "a result buffer that the allocator did not hand out");
  return nullptr;
}

PyObject* type_member(int t) { return t >= 0 && t <= B2_STRUCT && type_ids[t] ? type_ids[t] : Py_None; }

PyObject* as_column(b2_owned_column& c, Buffers& b)
{
  const size_t w = (size_t)width_of(c.type_id);
  const size_t data_used = w ? std::max<size_t>(((size_t)c.size * w + 3) / 4 * 4, 8) : 0;
  const size_t mask_used = std::max<size_t>(1, ((size_t)c.size + 511) / 512) * 64;
  Ref data(as_tensor(b, c.data, data_used));
  void* m = c.null_mask;
  Ref mask(as_tensor(b, m, mask_used));
  c.null_mask = (uint32_t*)m;
  if (!data.p || !mask.p) return nullptr;
  Ref offsets(nullptr), kids(nullptr);
  int offsets_type = B2_INT32;
  if (c.type_id == B2_STRUCT || c.type_id == B2_DICTIONARY32) {
    kids.p = PyList_New(c.num_children);
    for (int i = 0; kids.p && i < c.num_children; ++i) {
      PyObject* k = as_column(c.children[i], b);
      if (!k) return nullptr;
      PyList_SET_ITEM(kids.p, i, k);
    }
    if (!kids.p) return nullptr;
  } else if (c.num_children) {
    offsets.p = as_tensor(b, c.children[0].data, 0);
    offsets_type = c.children[0].type_id;
    if (!offsets.p) return nullptr;
  }
  return PyObject_CallFunction(fn_adopt, "OiOOiOOiO", type_member(c.type_id), (int)c.size, data.p, mask.p, (int)c.null_count,
                               offsets.p ? offsets.p : Py_None, type_member(offsets_type), (int)c.scale, kids.p ? kids.p : Py_None);
}

PyObject* as_table(b2_owned_column* cols, int n, Buffers& b)
{
  Ref list(PyList_New(n));
  if (!list.p) return nullptr;
  for (int i = 0; i < n; ++i) {
    PyObject* c = as_column(cols[i], b);
    if (!c) return nullptr;
    PyList_SET_ITEM(list.p, i, c);
  }
  return PyObject_CallOneArg(cls_table, list.p);
}

PyObject* as_result(b2_groupby_result& res, Buffers& b)
{
  PyObject* out = nullptr;
  Ref keys(as_table(res.keys, res.num_keys, b));
  if (keys.p) {
    Ref list(PyList_New(res.num_requests));
    bool ok = list.p != nullptr;
    for (int q = 0; ok && q < res.num_requests; ++q) {
      PyObject* t = as_table(res.results[q], res.num_results[q], b);
      ok = t != nullptr;
      if (ok) PyList_SET_ITEM(list.p, q, t);
    }
    if (ok) out = PyTuple_Pack(2, keys.p, list.p);
  }
  b2_result_free(&res);
  return out;
}

// a failed call: the package's _check raises the exception of the status
PyObject* fail(b2_status s)
{
  Ref r(PyObject_CallFunction(fn_check, "i", (int)s));
  if (r.p && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "the library reported a failure");
  return nullptr;
}

// where a call runs: the device of its columns (or the current one) and torch's current stream there
struct Place {
  c10::cuda::OptionalCUDAGuard guard;
  void* stream = nullptr;
  explicit Place(int device)
  {
    if (device >= 0) guard.set_index((c10::DeviceIndex)device);
    stream = c10::cuda::getCurrentCUDAStream().stream();
  }
};

template <typename F>
PyObject* wrapped(F&& f)
{
  try {
    return f();
  } catch (const PyFailed&) {
    return nullptr;
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// ------------------------------------------------------------------------------ module functions
PyObject* m_setup(PyObject*, PyObject* args)
{
  PyObject* ids;
  if (!PyArg_ParseTuple(args, "OOOO", &cls_table, &fn_adopt, &fn_check, &ids)) return nullptr;
  Py_INCREF(cls_table); Py_INCREF(fn_adopt); Py_INCREF(fn_check);
  Ref fast(PySequence_Fast(ids, "type ids"));
  if (!fast.p) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(fast.p); ++i) {
    PyObject* t = PySequence_Fast_GET_ITEM(fast.p, i);
    const long v = PyLong_AsLong(t);
    if (v >= 0 && v <= B2_STRUCT) { Py_INCREF(t); type_ids[v] = t; }
  }
  Py_RETURN_NONE;
}

// create(key columns, null policy, expected groups, table variant, shared table bytes, row filter columns) -> (handle, device index or -1)
PyObject* m_create(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 6) { PyErr_SetString(PyExc_TypeError, "create takes 6 arguments"); return nullptr; }
    Ref cols(PySequence_Fast(args[0], "keys is not a sequence")), filt(PySequence_Fast(args[5], "filters is not a sequence"));
    if (!cols.p || !filt.p) return nullptr;
    Kids kids;
    int device = -1;
    std::vector<b2_column_view> views;
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(cols.p); ++i)
      views.push_back(view_of(PySequence_Fast_GET_ITEM(cols.p, i), kids, &device));
    b2_groupby_options o{};
    o.expected_groups = PyLong_AsLongLong(args[2]);
    o.table_variant = (int32_t)PyLong_AsLong(args[3]);
    o.shared_table_bytes = (int32_t)PyLong_AsLong(args[4]);
    const int policy = (int)PyLong_AsLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    std::vector<const uint32_t*> masks;
    std::vector<int32_t> offsets;
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(filt.p); ++i) {
      PyObject* c = PySequence_Fast_GET_ITEM(filt.p, i);
      const uint32_t* m = (const uint32_t*)tensor_attr(c, n_mask, nullptr, nullptr);
      if (!m) continue;
      masks.push_back(m);
      offsets.push_back((int32_t)int_attr(c, n_offset));
    }
    o.num_row_filters = (int32_t)masks.size();
    o.row_filter_masks = masks.data();
    o.row_filter_offsets = offsets.data();
    b2_groupby* gb = nullptr;
    const b2_status s = b2_groupby_create(views.data(), (int32_t)views.size(), policy, &o, &gb);
    if (s != B2_SUCCESS) return fail(s);
    Ref handle(PyLong_FromVoidPtr(gb)), dev(PyLong_FromLong(device));
    return handle.p && dev.p ? PyTuple_Pack(2, handle.p, dev.p) : nullptr;
  });
}

PyObject* m_destroy(PyObject*, PyObject* h)
{
  void* p = PyLong_AsVoidPtr(h);
  if (!p && PyErr_Occurred()) return nullptr;
  b2_groupby_destroy((b2_groupby*)p);
  Py_RETURN_NONE;
}

// aggregate(handle, requests, device index or -1) -> (keys table, [table per request])
PyObject* m_aggregate(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "aggregate takes 3 arguments"); return nullptr; }
    b2_groupby* gb = (b2_groupby*)PyLong_AsVoidPtr(args[0]);
    int device = (int)PyLong_AsLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    Kids kids;
    Requests rq;
    read_requests(args[1], rq, kids, &device);
    Place at(device);
    Buffers bufs;
    bufs.live.reserve(16);
    b2_allocator al{take_buffer, give_buffer, &bufs};
    b2_groupby_result res{};
    b2_status s;
    Py_BEGIN_ALLOW_THREADS
    s = b2_groupby_aggregate(gb, rq.reqs.data(), (int32_t)rq.reqs.size(), at.stream, &al, &res);
    Py_END_ALLOW_THREADS
    return s == B2_SUCCESS ? as_result(res, bufs) : fail(s);
  });
}

// state_update(state, groupby handle, requests, device)
PyObject* m_state_update(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 4) { PyErr_SetString(PyExc_TypeError, "state_update takes 4 arguments"); return nullptr; }
    b2_groupby_state* st = (b2_groupby_state*)PyLong_AsVoidPtr(args[0]);
    b2_groupby* gb = (b2_groupby*)PyLong_AsVoidPtr(args[1]);
    int device = (int)PyLong_AsLong(args[3]);
    if (PyErr_Occurred()) return nullptr;
    Kids kids;
    Requests rq;
    read_requests(args[2], rq, kids, &device);
    Place at(device);
    b2_status s;
    Py_BEGIN_ALLOW_THREADS
    s = b2_state_update(st, gb, rq.reqs.data(), (int32_t)rq.reqs.size(), at.stream);
    Py_END_ALLOW_THREADS
    if (s != B2_SUCCESS) return fail(s);
    Py_RETURN_NONE;
  });
}

// state_create(groupby handle, requests) -> handle
PyObject* m_state_create(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "state_create takes 2 arguments"); return nullptr; }
    b2_groupby* gb = (b2_groupby*)PyLong_AsVoidPtr(args[0]);
    if (PyErr_Occurred()) return nullptr;
    Kids kids;
    Requests rq;
    read_requests(args[1], rq, kids, nullptr);
    b2_groupby_state* st = nullptr;
    const b2_status s = b2_state_create(gb, rq.reqs.data(), (int32_t)rq.reqs.size(), &st);
    return s == B2_SUCCESS ? PyLong_FromVoidPtr(st) : fail(s);
  });
}

PyObject* m_state_num_groups(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "state_num_groups takes 2 arguments"); return nullptr; }
    b2_groupby_state* st = (b2_groupby_state*)PyLong_AsVoidPtr(args[0]);
    const int device = (int)PyLong_AsLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    Place at(device);
    int64_t n = 0;
    b2_status s;
    Py_BEGIN_ALLOW_THREADS
    s = b2_state_num_groups(st, at.stream, &n);
    Py_END_ALLOW_THREADS
    return s == B2_SUCCESS ? PyLong_FromLongLong(n) : fail(s);
  });
}

PyObject* m_state_finalize(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "state_finalize takes 2 arguments"); return nullptr; }
    b2_groupby_state* st = (b2_groupby_state*)PyLong_AsVoidPtr(args[0]);
    const int device = (int)PyLong_AsLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    Place at(device);
    Buffers bufs;
    b2_allocator al{take_buffer, give_buffer, &bufs};
    b2_groupby_result res{};
    b2_status s;
    Py_BEGIN_ALLOW_THREADS
    s = b2_state_finalize(st, at.stream, &al, &res);
    Py_END_ALLOW_THREADS
    return s == B2_SUCCESS ? as_result(res, bufs) : fail(s);
  });
}

// hash_partition(columns with the hashed ones first, number hashed, parts, hash function, seed, device) -> ([column], [offset])
PyObject* m_hash_partition(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
  return wrapped([&]() -> PyObject* {
    if (nargs != 6) { PyErr_SetString(PyExc_TypeError, "hash_partition takes 6 arguments"); return nullptr; }
    const int nhash = (int)PyLong_AsLong(args[1]);
    const long parts = PyLong_AsLong(args[2]);
    const int kind = (int)PyLong_AsLong(args[3]);
    const uint32_t seed = (uint32_t)PyLong_AsUnsignedLong(args[4]);
    int device = (int)PyLong_AsLong(args[5]);
    if (PyErr_Occurred()) return nullptr;
    Ref cols(PySequence_Fast(args[0], "columns is not a sequence"));
    if (!cols.p) return nullptr;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(cols.p);
    Kids kids;
    std::vector<b2_column_view> views;
    for (Py_ssize_t i = 0; i < n; ++i) views.push_back(view_of(PySequence_Fast_GET_ITEM(cols.p, i), kids, &device));
    Place at(device);
    Buffers bufs;
    b2_allocator al{take_buffer, give_buffer, &bufs};
    std::vector<b2_owned_column> out((size_t)n + 1);
    std::vector<int64_t> offsets((size_t)(parts < 0 ? 0 : parts) + 1);
    b2_status s;
    Py_BEGIN_ALLOW_THREADS
    s = b2_hash_partition(views.data(), (int32_t)n, nhash, (int32_t)parts, kind, seed, at.stream, &al, out.data(), offsets.data());
    Py_END_ALLOW_THREADS
    if (s != B2_SUCCESS) return fail(s);
    Ref list(PyList_New(n)), offs(PyList_New((Py_ssize_t)offsets.size()));
    bool ok = list.p && offs.p;
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* c = ok ? as_column(out[(size_t)i], bufs) : nullptr;
      if (c) PyList_SET_ITEM(list.p, i, c); else ok = false;
      b2_column_free(&out[(size_t)i], &al, at.stream);  // the host arrays of the descriptor
    }
    for (size_t p = 0; ok && p < offsets.size(); ++p) PyList_SET_ITEM(offs.p, (Py_ssize_t)p, PyLong_FromLongLong(offsets[p]));
    return ok ? PyTuple_Pack(2, list.p, offs.p) : nullptr;
  });
}

#define FAST(name) #name, (PyCFunction)(void (*)(void))m_##name, METH_FASTCALL, nullptr
PyMethodDef methods[] = {
  {"setup", m_setup, METH_VARARGS, nullptr},
  {FAST(create)},
  {"destroy", m_destroy, METH_O, nullptr},
  {FAST(aggregate)},
  {FAST(state_create)},
  {FAST(state_update)},
  {FAST(state_num_groups)},
  {FAST(state_finalize)},
  {FAST(hash_partition)},
  {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b2native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b2native(void)
{
  struct { PyObject** slot; const char* name; } names[] = {
    {&n_type_id, "type_id"}, {&n_scale, "scale"}, {&n_size, "size"}, {&n_null_count, "null_count"}, {&n_data, "data"}, {&n_mask, "mask"},
    {&n_offset, "offset"}, {&n_offsets, "offsets"}, {&n_offsets_type, "offsets_type"}, {&n_children, "children"}, {&n_values, "_values"},
    {&n_aggregations, "_aggregations"}, {&n_kind, "kind"}, {&n_ddof, "ddof"}};
  for (auto& n : names)
    if (!(*n.slot = PyUnicode_InternFromString(n.name))) return nullptr;
  return PyModule_Create(&module);
}
