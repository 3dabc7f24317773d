// CPython binding of the tensor-level entry points (habitat_b200/batched.py).
//
// A small launch is bound by the host: through ctypes, wave_scale spent 45 us on argument objects, five
// allocations, device look-ups and structure building for a kernel of 5 us.  This module reads the torch
// tensors directly, makes small results in one allocation and calls the C ABI through function addresses
// that _native.py hands over (so that another build of the library can stand in).  It holds no arithmetic
// and no state but those addresses.  Every argument is checked as batched.py documents; a check that fails
// makes the function return None, and the caller's Python checks then raise the error.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "habitat_b200.h"

namespace {

struct Api {
  decltype(&hb_wave_scale) wave_scale = nullptr;
  decltype(&hb_wave_scale_metrics) wave_scale_metrics = nullptr;
  decltype(&hb_wave_scale_partials) wave_scale_partials = nullptr;
  decltype(&hb_partials_sum) partials_sum = nullptr;
  decltype(&hb_mlp_predict) mlp_predict = nullptr;
  decltype(&hb_mlp_predict_host) mlp_predict_host = nullptr;
  decltype(&hb_group_sum) group_sum = nullptr;
  decltype(&hb_plane_sum) plane_sum = nullptr;
  decltype(&hb_segment_sum) segment_sum = nullptr;
} api;

PyObject* g_row_of = nullptr;       // device_table.row_of
PyObject* g_raise = nullptr;        // _native.check
PyObject* g_wave_result = nullptr;  // batched.WaveResult
long g_generation = 0;              // of the device table; tokens of an older one are looked up again

PyObject *s_num_blocks, *s_block_size, *s_regs, *s_smem, *s_time, *s_gamma, *s_row_token, *s_flop, *s_rd, *s_wr,
    *s_has, *s_scaled, *s_docc, *s_dwav, *s_oocc, *s_owav, *s_status, *s_limits, *s_buffer, *s_K, *s_D, *s_per_plane,
    *s_n_planes;

// A reference that is dropped at the end of the scope.
struct Ref {
  PyObject* p;
  explicit Ref(PyObject* q) : p(q) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
};

// The data of a contiguous CUDA tensor of `type`; null when `o` is anything else.
const at::Tensor* tensor(PyObject* o, at::ScalarType type) {
  if (!o || !THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.scalar_type() == type && t.is_contiguous() ? &t : nullptr;
}
void* data(const at::Tensor* t) { return t ? t->mutable_data_ptr() : nullptr; }

// Attribute `name` of `o` as tensor data; the tensor stays alive through its owner.
struct Field {
  Ref ref;
  const at::Tensor* t;
  Field(PyObject* o, PyObject* name, at::ScalarType type) : ref(PyObject_GetAttr(o, name)), t(nullptr) {
    if (!ref.p) PyErr_Clear();
    else t = tensor(ref.p, type);
  }
  bool none() const { return ref.p == Py_None; }
  void* ptr() const { return data(t); }
};

// Row of a DeviceProperties in the library's table: its token (generation * 64 + row) when it is of the
// current table, else device_table.row_of.  -1 with a Python error set when that fails.
long row_of(PyObject* device) {
  Ref token(PyObject_GetAttr(device, s_row_token));
  if (token.p && PyLong_Check(token.p)) {
    const long v = PyLong_AsLong(token.p);
    if (v >= 0 && v / HB_MAX_DEVICES == g_generation) return v % HB_MAX_DEVICES;
  }
  PyErr_Clear();
  Ref row(PyObject_CallOneArg(g_row_of, device));
  if (!row.p) return -1;
  return PyLong_AsLong(row.p);
}

bool failed(hb_status st) {
  if (st == HB_OK) return false;
  Ref code(PyLong_FromLong(st));
  Ref r(PyObject_CallOneArg(g_raise, code.p));   // raises HabitatNativeError with the library's text
  if (r.p && !PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "native call failed");
  return true;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) {
  return at::Tensor(at::detail::empty_cuda(sizes, type, dev, c10::nullopt));
}
// A contiguous tensor of `type` at byte `offset` of another one's storage.
at::Tensor inside(const at::Tensor& block, size_t offset, at::IntArrayRef sizes, at::ScalarType type) {
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(block.storage()),
                                                          c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                          c10::scalarTypeToTypeMeta(type));
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  t.unsafeGetTensorImpl()->set_storage_offset(static_cast<int64_t>(offset / c10::elementSize(type)));
  return t;
}

// Results up to this size share one allocation (each plane on a 256-byte boundary): an allocation costs
// about a microsecond.  Larger ones are separate, so that a caller who keeps one plane keeps only that.
constexpr size_t kOneBlock = 1 << 20;

hb_status wave_scale_call(const hb_kernel_soa& k, const hb_kernel_metrics* m, int64_t K, int32_t origin,
                          const int32_t* rows, int32_t D, const int16_t* regs, const hb_wave_out& out, double* partials,
                          int32_t* per_plane, void* stream) {
  hb_status st;
  Py_BEGIN_ALLOW_THREADS
  if (partials) st = api.wave_scale_partials(&k, K, origin, rows, D, regs, &out, partials, per_plane, stream);
  else if (m) st = api.wave_scale_metrics(&k, m, K, origin, rows, D, regs, &out, stream);
  else st = api.wave_scale(&k, K, origin, rows, D, regs, &out, stream);
  Py_END_ALLOW_THREADS
  return st;
}

// wave_scale(kernels, origin, dests, dest_regs, metrics, want_status, want_limits, out, partials)
PyObject* wave_scale(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9) Py_RETURN_NONE;
  PyObject *kernels = a[0], *metrics = a[4], *out = a[7], *partials = a[8];
  const Field nb(kernels, s_num_blocks, at::kInt), bs(kernels, s_block_size, at::kUInt16),
      rg(kernels, s_regs, at::kUInt16), sm(kernels, s_smem, at::kUInt32), tm(kernels, s_time, at::kFloat),
      gm(kernels, s_gamma, at::kFloat);
  if (!nb.t || !bs.t || !rg.t || !sm.t || !tm.t || (metrics == Py_None && !gm.t)) Py_RETURN_NONE;
  const int64_t K = nb.t->numel();
  if (bs.t->numel() != K || rg.t->numel() != K || sm.t->numel() != K || tm.t->numel() != K) Py_RETURN_NONE;

  Ref dests(PySequence_Fast(a[2], "dests must be a sequence of DeviceProperties"));
  if (!dests.p) return nullptr;
  const Py_ssize_t D = PySequence_Fast_GET_SIZE(dests.p);
  if (D > HB_MAX_DEVICES) Py_RETURN_NONE;
  int32_t rows[HB_MAX_DEVICES];
  const long origin = row_of(a[1]);
  if (origin < 0) return nullptr;
  for (Py_ssize_t d = 0; d < D; ++d) {
    const long r = row_of(PySequence_Fast_GET_ITEM(dests.p, d));
    if (r < 0) return nullptr;
    rows[d] = static_cast<int32_t>(r);
  }

  const int16_t* regs = nullptr;
  if (a[3] != Py_None) {
    const at::Tensor* t = tensor(a[3], at::kShort);
    if (!t || t->dim() != 2 || t->size(0) != D || t->size(1) != K) Py_RETURN_NONE;
    regs = static_cast<const int16_t*>(data(t));
  }
  hb_kernel_metrics m{};
  if (metrics != Py_None) {
    if (partials != Py_None) Py_RETURN_NONE;
    const Field fe(metrics, s_flop, at::kDouble), rd(metrics, s_rd, at::kDouble), wr(metrics, s_wr, at::kDouble),
        has(metrics, s_has, at::kByte);
    if (!fe.t || !rd.t || !wr.t || !has.t) Py_RETURN_NONE;
    m.flop_efficiency_pct = static_cast<const double*>(fe.ptr());
    m.dram_read_bytes = static_cast<const double*>(rd.ptr());
    m.dram_write_bytes = static_cast<const double*>(wr.ptr());
    m.has_metrics = static_cast<const uint8_t*>(has.ptr());
  }
  double* sums = nullptr;
  if (partials != Py_None) {
    Ref pk(PyObject_GetAttr(partials, s_K)), pd(PyObject_GetAttr(partials, s_D));
    const Field buf(partials, s_buffer, at::kDouble);
    if (!pk.p || !pd.p || !buf.t || K > PyLong_AsLongLong(pk.p) || D > PyLong_AsLongLong(pd.p)) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    sums = static_cast<double*>(buf.ptr());
  }

  hb_kernel_soa k{static_cast<const int32_t*>(nb.ptr()), static_cast<const uint16_t*>(bs.ptr()),
                  static_cast<const uint16_t*>(rg.ptr()), static_cast<const uint32_t*>(sm.ptr()),
                  static_cast<const float*>(tm.ptr()), static_cast<const float*>(gm.ptr())};
  hb_wave_out o{};
  Ref made(nullptr);
  if (out == Py_None) {
    const bool status = PyObject_IsTrue(a[5]) == 1, limits = PyObject_IsTrue(a[6]) == 1;
    const at::Device dev = nb.t->device();
    const int64_t dk[2] = {D, K}, k1[1] = {K}, lim[3] = {D + 1, 4, K};
    struct Plane { at::IntArrayRef sizes; at::ScalarType type; size_t bytes; bool want; };
    const size_t pairs = static_cast<size_t>(D) * K, kk = static_cast<size_t>(K);
    const Plane planes[7] = {{dk, at::kFloat, pairs * 4, true},  {dk, at::kByte, pairs, true},
                             {dk, at::kUInt32, pairs * 4, true}, {k1, at::kByte, kk, true},
                             {k1, at::kUInt32, kk * 4, true},    {dk, at::kByte, pairs, status},
                             {lim, at::kInt, 16 * (D + 1) * kk, limits}};
    size_t offset[7], total = 0;
    for (int i = 0; i < 7; ++i) {
      offset[i] = total;
      if (planes[i].want) total += (planes[i].bytes + 255) & ~static_cast<size_t>(255);
    }
    const bool one = total <= kOneBlock;
    at::Tensor block;
    if (one) {
      const int64_t size[1] = {static_cast<int64_t>(total)};
      block = empty(size, at::kByte, dev);
    }
    void* ptr[7];
    PyObject* args[8] = {nullptr};
    for (int i = 0; i < 7; ++i) {
      ptr[i] = nullptr;
      if (!planes[i].want) {
        args[1 + i] = Py_NewRef(Py_None);
        continue;
      }
      at::Tensor t = one ? inside(block, offset[i], planes[i].sizes, planes[i].type)
                         : empty(planes[i].sizes, planes[i].type, dev);
      ptr[i] = t.mutable_data_ptr();
      args[1 + i] = THPVariable_Wrap(std::move(t));
    }
    made.p = PyObject_Vectorcall(g_wave_result, args + 1, 7 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    for (int i = 0; i < 7; ++i) Py_XDECREF(args[1 + i]);
    if (!made.p) return nullptr;
    o = hb_wave_out{static_cast<float*>(ptr[0]),    static_cast<uint8_t*>(ptr[1]),  static_cast<uint32_t*>(ptr[2]),
                    static_cast<uint8_t*>(ptr[3]),  static_cast<uint32_t*>(ptr[4]), static_cast<uint8_t*>(ptr[5]),
                    static_cast<int32_t*>(ptr[6])};
  } else {
    // given results are taken as they are (their pointers), like the planes of any earlier call
    PyObject* names[7] = {s_scaled, s_docc, s_dwav, s_oocc, s_owav, s_status, s_limits};
    void* ptr[7];
    for (int i = 0; i < 7; ++i) {
      Ref f(PyObject_GetAttr(out, names[i]));
      if (!f.p) return nullptr;
      if (f.p != Py_None && !THPVariable_Check(f.p)) Py_RETURN_NONE;
      ptr[i] = f.p == Py_None ? nullptr : THPVariable_Unpack(f.p).mutable_data_ptr();
    }
    o = hb_wave_out{static_cast<float*>(ptr[0]),    static_cast<uint8_t*>(ptr[1]),  static_cast<uint32_t*>(ptr[2]),
                    static_cast<uint8_t*>(ptr[3]),  static_cast<uint32_t*>(ptr[4]), static_cast<uint8_t*>(ptr[5]),
                    static_cast<int32_t*>(ptr[6])};
    made.p = Py_NewRef(out);
  }
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  int32_t per_plane = 0;
  const hb_status st = wave_scale_call(k, metrics == Py_None ? nullptr : &m, K, static_cast<int32_t>(origin), rows,
                                       static_cast<int32_t>(D), regs, o, sums, &per_plane, stream);
  if (sums) {
    Ref pp(PyLong_FromLong(per_plane)), np(PyLong_FromLong(static_cast<long>(D)));
    if (PyObject_SetAttr(partials, s_per_plane, pp.p) < 0 || PyObject_SetAttr(partials, s_n_planes, np.p) < 0)
      return nullptr;
  }
  if (failed(st)) return nullptr;
  PyObject* result = made.p;
  made.p = nullptr;
  return result;
  END_HANDLE_TH_ERRORS
}

// The optional `out` argument of a sum: itself when it fits, a new tensor for None, undefined otherwise.
at::Tensor sum_out(PyObject* o, int64_t n, const at::Device& dev) {
  if (o == Py_None) {
    const int64_t size[1] = {n};
    return empty(size, at::kDouble, dev);
  }
  const at::Tensor* t = tensor(o, at::kDouble);
  return t && t->numel() == n ? *t : at::Tensor();
}
PyObject* sum_result(PyObject* o, at::Tensor&& t) { return o == Py_None ? THPVariable_Wrap(std::move(t)) : Py_NewRef(o); }

// mlp_predict(handle address, F, op_features, device_row, out)
PyObject* mlp_predict(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) Py_RETURN_NONE;
  hb_mlp* h = static_cast<hb_mlp*>(PyLong_AsVoidPtr(a[0]));
  const long F = PyLong_AsLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor *f = tensor(a[2], at::kFloat), *r = tensor(a[3], at::kByte);
  if (!f || !r || f->dim() != 2 || f->size(1) != F || r->numel() != f->size(0)) Py_RETURN_NONE;
  const int64_t Q = f->size(0);
  at::Tensor made;
  void* out;
  if (a[4] == Py_None) {
    const int64_t size[1] = {Q};
    made = empty(size, at::kFloat, f->device());
    out = made.mutable_data_ptr();
  } else {
    if (!THPVariable_Check(a[4])) Py_RETURN_NONE;
    out = THPVariable_Unpack(a[4]).mutable_data_ptr();
  }
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  const float* pf = static_cast<const float*>(data(f));
  const uint8_t* pr = static_cast<const uint8_t*>(data(r));
  hb_status st;
  Py_BEGIN_ALLOW_THREADS
  st = api.mlp_predict(h, pf, pr, Q, static_cast<float*>(out), stream);
  Py_END_ALLOW_THREADS
  if (failed(st)) return nullptr;
  return a[4] == Py_None ? THPVariable_Wrap(std::move(made)) : Py_NewRef(a[4]);
  END_HANDLE_TH_ERRORS
}

// mlp_predict_one(handle address, F, op features of one query, device row) -> float
PyObject* mlp_predict_one(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) Py_RETURN_NONE;
  hb_mlp* h = static_cast<hb_mlp*>(PyLong_AsVoidPtr(a[0]));
  const long F = PyLong_AsLong(a[1]), row = PyLong_AsLong(a[3]);
  Ref seq(PySequence_Fast(a[2], "the operation's features must be a sequence"));
  if (!seq.p || PyErr_Occurred()) return nullptr;
  constexpr long kMaxF = 8;
  if (F > kMaxF || PySequence_Fast_GET_SIZE(seq.p) != F || row < 0 || row > 255) Py_RETURN_NONE;
  float f[kMaxF], out = 0.0f;
  for (long i = 0; i < F; ++i) {
    const double v = PyFloat_AsDouble(PySequence_Fast_GET_ITEM(seq.p, i));
    if (v == -1.0 && PyErr_Occurred()) return nullptr;
    f[i] = static_cast<float>(v);
  }
  const uint8_t r = static_cast<uint8_t>(row);
  hb_status st;
  Py_BEGIN_ALLOW_THREADS
  st = api.mlp_predict_host(h, f, &r, 1, &out);
  Py_END_ALLOW_THREADS
  if (failed(st)) return nullptr;
  return PyFloat_FromDouble(out);
}

// partials_sum(buffer, per_plane, n_planes, out)
PyObject* partials_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) Py_RETURN_NONE;
  const at::Tensor* buf = tensor(a[0], at::kDouble);
  const long per_plane = PyLong_AsLong(a[1]), planes = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (!buf) Py_RETURN_NONE;
  at::Tensor out = sum_out(a[3], planes, buf->device());
  if (!out.defined()) Py_RETURN_NONE;
  if (failed(api.partials_sum(static_cast<const double*>(data(buf)), static_cast<int32_t>(per_plane),
                              static_cast<int32_t>(planes), static_cast<double*>(out.mutable_data_ptr()),
                              c10::cuda::getCurrentCUDAStream().stream())))
    return nullptr;
  return sum_result(a[3], std::move(out));
  END_HANDLE_TH_ERRORS
}

// group_sum(values, keys, n_groups, out)
PyObject* group_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) Py_RETURN_NONE;
  const at::Tensor *v = tensor(a[0], at::kFloat), *k = tensor(a[1], at::kByte);
  const long groups = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (!v || !k || v->numel() != k->numel() || groups < 0) Py_RETURN_NONE;
  at::Tensor out = sum_out(a[3], groups, v->device());
  if (!out.defined()) Py_RETURN_NONE;
  if (failed(api.group_sum(static_cast<const float*>(data(v)), static_cast<const uint8_t*>(data(k)), v->numel(),
                           static_cast<int32_t>(groups), static_cast<double*>(out.mutable_data_ptr()),
                           c10::cuda::getCurrentCUDAStream().stream())))
    return nullptr;
  return sum_result(a[3], std::move(out));
  END_HANDLE_TH_ERRORS
}

// plane_sum(values, out)
PyObject* plane_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) Py_RETURN_NONE;
  const at::Tensor* v = tensor(a[0], at::kFloat);
  if (!v || v->dim() != 2) Py_RETURN_NONE;
  at::Tensor out = sum_out(a[1], v->size(0), v->device());
  if (!out.defined()) Py_RETURN_NONE;
  if (failed(api.plane_sum(static_cast<const float*>(data(v)), v->size(1), static_cast<int32_t>(v->size(0)),
                           static_cast<double*>(out.mutable_data_ptr()), c10::cuda::getCurrentCUDAStream().stream())))
    return nullptr;
  return sum_result(a[1], std::move(out));
  END_HANDLE_TH_ERRORS
}

// segment_sum(values, offsets)
PyObject* segment_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) Py_RETURN_NONE;
  const at::Tensor *v = tensor(a[0], at::kFloat), *o = tensor(a[1], at::kLong);
  if (!v || !o) Py_RETURN_NONE;
  const int64_t segments = o->numel() - 1;
  at::Tensor out = sum_out(Py_None, segments > 0 ? segments : 0, v->device());
  if (failed(api.segment_sum(static_cast<const float*>(data(v)), static_cast<const int64_t*>(data(o)), segments,
                             static_cast<double*>(out.mutable_data_ptr()), c10::cuda::getCurrentCUDAStream().stream())))
    return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// setup(addresses by name, row_of, check, WaveResult)
PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4 || !PyDict_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "setup(addresses, row_of, check, WaveResult)");
    return nullptr;
  }
  auto load = [&](auto& fn, const char* name) {
    PyObject* v = PyDict_GetItemString(a[0], name);   // borrowed
    fn = v ? reinterpret_cast<std::remove_reference_t<decltype(fn)>>(PyLong_AsVoidPtr(v)) : nullptr;
    return fn != nullptr;
  };
  if (!load(api.wave_scale, "hb_wave_scale") || !load(api.wave_scale_metrics, "hb_wave_scale_metrics") ||
      !load(api.wave_scale_partials, "hb_wave_scale_partials") || !load(api.partials_sum, "hb_partials_sum") ||
      !load(api.mlp_predict, "hb_mlp_predict") || !load(api.mlp_predict_host, "hb_mlp_predict_host") || !load(api.group_sum, "hb_group_sum") ||
      !load(api.plane_sum, "hb_plane_sum") || !load(api.segment_sum, "hb_segment_sum")) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "an entry point is missing");
    return nullptr;
  }
  Py_XSETREF(g_row_of, Py_NewRef(a[1]));
  Py_XSETREF(g_raise, Py_NewRef(a[2]));
  Py_XSETREF(g_wave_result, Py_NewRef(a[3]));
  Py_RETURN_NONE;
}

PyObject* set_generation(PyObject*, PyObject* v) {
  g_generation = PyLong_AsLong(v);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(setup), FAST(wave_scale), FAST(mlp_predict), FAST(mlp_predict_one), FAST(partials_sum), FAST(group_sum),
                         FAST(plane_sum), FAST(segment_sum),
                         {"set_generation", set_generation, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) {
  const struct { PyObject** s; const char* name; } names[] = {
      {&s_num_blocks, "num_blocks"}, {&s_block_size, "block_size"}, {&s_regs, "regs_per_thread"},
      {&s_smem, "smem_bytes"}, {&s_time, "run_time_ns"}, {&s_gamma, "gamma"}, {&s_row_token, "_row_token"},
      {&s_flop, "flop_efficiency_pct"}, {&s_rd, "dram_read_bytes"}, {&s_wr, "dram_write_bytes"},
      {&s_has, "has_metrics"}, {&s_scaled, "scaled_ns"}, {&s_docc, "dest_occupancy"}, {&s_dwav, "dest_waves"},
      {&s_oocc, "origin_occupancy"}, {&s_owav, "origin_waves"}, {&s_status, "status"}, {&s_limits, "limits"},
      {&s_buffer, "buffer"}, {&s_K, "K"}, {&s_D, "D"}, {&s_per_plane, "per_plane"}, {&s_n_planes, "n_planes"}};
  for (const auto& n : names)
    if (!(*n.s = PyUnicode_InternFromString(n.name))) return nullptr;
  return PyModule_Create(&module);
}
