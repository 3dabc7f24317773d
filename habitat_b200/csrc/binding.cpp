// CPython binding of the tensor-level entry points (habitat_b200/batched.py).
//
// A small launch is bound by the host: through ctypes, wave_scale spent 45 us on argument objects, five
// allocations, device look-ups and structure building for a kernel of 5 us.  This module reads the torch
// tensors directly, makes small results in one allocation and calls the C ABI through function addresses
// that _native.py hands over (so that another build of the library can stand in).  Its state is those addresses
// and the pool of page-locked blocks for host results.  Every argument is checked as batched.py documents; a check
// that fails makes the function return None, and the caller's Python checks then raise the error.
#include <Python.h>

#include <ATen/EmptyTensor.h>
#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime_api.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "habitat_b200.h"

namespace {

struct Api {
  decltype(&hb_wave_scale) wave_scale = nullptr;
  decltype(&hb_wave_scale_metrics) wave_scale_metrics = nullptr;
  decltype(&hb_wave_scale_partials) wave_scale_partials = nullptr;
  decltype(&hb_wave_scale_host) wave_scale_host = nullptr;
  decltype(&hb_partials_sum) partials_sum = nullptr;
  decltype(&hb_mlp_predict) mlp_predict = nullptr;
  decltype(&hb_mlp_predict_host) mlp_predict_host = nullptr;
  decltype(&hb_group_sum) group_sum = nullptr;
  decltype(&hb_plane_sum) plane_sum = nullptr;
  decltype(&hb_segment_sum) segment_sum = nullptr;
  decltype(&hb_segment_sum_planes) segment_sum_planes = nullptr;
  decltype(&hb_mlp_predict_grid) mlp_predict_grid = nullptr;
  decltype(&hb_mlp_poll_status) mlp_poll_status = nullptr;
  decltype(&hb_special_scale_grid) special_scale_grid = nullptr;
  decltype(&hb_iteration_totals) iteration_totals = nullptr;
} api;

PyObject* g_row_of = nullptr;       // device_table.row_of
PyObject* g_raise = nullptr;        // _native.check
PyObject* g_wave_result = nullptr;  // batched.WaveResult
PyObject* g_device_type = nullptr;  // habitat_cuda.DeviceProperties
long g_generation = 0;              // of the device table; tokens of an older one are looked up again

PyObject *s_num_blocks, *s_block_size, *s_regs, *s_smem, *s_time, *s_gamma, *s_row_token, *s_flop, *s_rd, *s_wr,
    *s_has, *s_scaled, *s_docc, *s_dwav, *s_oocc, *s_owav, *s_status, *s_limits, *s_buffer, *s_K, *s_D, *s_per_plane,
    *s_n_planes, *s__name, *s__device, *s__forward, *s__backward, *s__arguments, *s_args, *s_kwargs, *s__kernels,
    *s__run_time_ms, *s__c, *s__metrics_kernels, *s__cached_metrics, *s__metrics, *s__num_blocks, *s__block_size,
    *s__regs, *s__smem_static, *s__smem_dynamic, *s__run_time_ns, *s_name;

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
// A given result plane of at least `count` elements of `size` bytes that the GPU can write: its data, or null.
void* result_data(PyObject* o, size_t size, int64_t count) {
  if (!o || !THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return (t.is_cuda() || t.is_pinned()) && t.element_size() == size && t.is_contiguous() && t.numel() >= count
             ? t.mutable_data_ptr() : nullptr;
}

// Attribute `name` of `o` as tensor data; the tensor stays alive through its owner.
struct Field {
  Ref ref;
  const at::Tensor* t;
  Field(PyObject* o, PyObject* name, at::ScalarType type) : ref(PyObject_GetAttr(o, name)), t(nullptr) {
    if (!ref.p) PyErr_Clear();
    else t = tensor(ref.p, type);
  }
  void* ptr() const { return data(t); }
  bool covers(int64_t count) const { return t && t->numel() >= count; }
};

// Row of a device in the library's table: a DeviceProperties' token (generation * 64 + row) when it is of the
// current table, else device_table.row_of.  -1 with a Python error set when that fails.
long row_of(PyObject* device) {
  if (reinterpret_cast<PyObject*>(Py_TYPE(device)) == g_device_type) {
    Ref token(PyObject_GetAttr(device, s_row_token));
    if (token.p && PyLong_Check(token.p)) {
      const long v = PyLong_AsLong(token.p);
      if (v >= 0 && v / HB_MAX_DEVICES == g_generation) return v % HB_MAX_DEVICES;
    }
    PyErr_Clear();
  }
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
// The same beside tensors that are on the GPU already: with its device current, straight from torch's allocator
// (the general form looks up and switches devices, a tenth of a microsecond each time).
at::Tensor empty_beside(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev, bool current) {
  if (!current) return empty(sizes, type, dev);
  size_t bytes = c10::elementSize(type);
  for (const int64_t n : sizes) bytes *= static_cast<size_t>(n);
  c10::Allocator* allocator = c10::cuda::CUDACachingAllocator::get();
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(
      c10::Storage(c10::make_intrusive<c10::StorageImpl>(c10::StorageImpl::use_byte_size_t(), bytes, allocator->allocate(bytes),
                                                         allocator, /*resizable=*/true)),
      c10::DispatchKeySet(c10::DispatchKey::CUDA), c10::scalarTypeToTypeMeta(type));
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  return t;
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
// Only bytes and uint32 share: torch.save refuses tensors that see one storage as different types, and counts
// those two as one.
constexpr size_t kOneBlock = 1 << 20;
constexpr bool shares_block(at::ScalarType t) { return t == at::kByte || t == at::kUInt32; }

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
  if (!nb.t || !bs.t || !rg.t || !sm.t || !tm.t) Py_RETURN_NONE;
  const int64_t K = nb.t->numel();
  if (metrics == Py_None && !gm.covers(K)) Py_RETURN_NONE;
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
    if (!fe.covers(K) || !rd.covers(K) || !wr.covers(K) || !has.covers(K)) Py_RETURN_NONE;
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
      if (planes[i].want && shares_block(planes[i].type)) total += (planes[i].bytes + 255) & ~static_cast<size_t>(255);
    }
    const bool one = total <= kOneBlock, current = dev.index() == c10::cuda::current_device();
    at::Tensor block;
    if (one) {
      const int64_t size[1] = {static_cast<int64_t>(total)};
      block = empty_beside(size, at::kByte, dev, current);
    }
    void* ptr[7];
    PyObject* args[8] = {nullptr};
    for (int i = 0; i < 7; ++i) {
      ptr[i] = nullptr;
      if (!planes[i].want) {
        args[1 + i] = Py_NewRef(Py_None);
        continue;
      }
      at::Tensor t = one && shares_block(planes[i].type) ? inside(block, offset[i], planes[i].sizes, planes[i].type)
                                                         : empty_beside(planes[i].sizes, planes[i].type, dev, current);
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
    // given results: at least as large as this call's planes
    const int64_t dk = D * K, counts[7] = {dk, dk, dk, K, K, dk, (D + 1) * 4 * K};
    constexpr size_t kSizes[7] = {4, 1, 4, 1, 4, 1, 4};
    PyObject* names[7] = {s_scaled, s_docc, s_dwav, s_oocc, s_owav, s_status, s_limits};
    void* ptr[7];
    for (int i = 0; i < 7; ++i) {
      Ref f(PyObject_GetAttr(out, names[i]));
      if (!f.p) return nullptr;
      ptr[i] = f.p == Py_None ? nullptr : result_data(f.p, kSizes[i], counts[i]);
      if (f.p != Py_None && !ptr[i] && counts[i] > 0) Py_RETURN_NONE;
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
    out = result_data(a[4], 4, Q);
    if (!out && Q > 0) Py_RETURN_NONE;
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

// ---------------------------------------------------------------------------
// Traces (habitat_b200/analysis/predictor.py): the walk over recorded objects, and one prediction
// ---------------------------------------------------------------------------
// Attribute of an instance, new reference; null (with an error set) when it has none.
inline PyObject* get(PyObject* o, PyObject* name) { return PyObject_GetAttr(o, name); }
// The same for an instance of one of the package's recorded classes, which keep their fields in the instance:
// MeasuredKernel's __getattr__ makes the ordinary look-up go through a Python-level hook's slot.
inline PyObject* field(PyObject* o, PyObject* name) { return PyObject_GenericGetAttr(o, name); }
// The integer attribute `name`; *ok is cleared when it is not a 64-bit integer.
int64_t int_of(PyObject* o, PyObject* name, bool* ok) {
  Ref v(field(o, name));
  if (!v.p || !PyLong_Check(v.p)) {
    *ok = false;
    return 0;
  }
  const int64_t x = PyLong_AsLongLong(v.p);
  if (x == -1 && PyErr_Occurred()) *ok = false;
  return x;
}
PyObject* bytes_of(const void* p, size_t n) {
  return PyBytes_FromStringAndSize(static_cast<const char*>(p), static_cast<Py_ssize_t>(n));
}
template <typename T>
PyObject* bytes_of(const std::vector<T>& v) { return bytes_of(v.data(), v.size() * sizeof(T)); }
// "Not an ordinary trace": the caller takes the general path, which also raises what there is to raise.
PyObject* not_ordinary() {
  PyErr_Clear();
  Py_RETURN_NONE;
}
void* stream_now() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Mirrors MeasuredKernel.get_metric for the three metrics of the roofline rule, whose canonical value is the raw
// one.  The three metrics of a kernel ((Metric, name, legacy name) each) from the values it has looked up before or the
// first record that holds them: 1, 0 when one is missing, -1 (perhaps with an error set) when something is not of
// the ordinary classes.  One walk over the records; names are mostly the very objects that `metrics` holds.
int find_metrics(PyObject* records, PyObject* cached, PyObject* metrics, PyTypeObject* instance_type, double* out) {
  const Py_ssize_t n = PyList_GET_SIZE(records);
  if (n == 0 && PyDict_GET_SIZE(cached) == 0) return 0;
  PyObject* names[3][2];
  unsigned missing = 0;
  for (int m = 0; m < 3; ++m) {
    PyObject* t = PyTuple_GET_ITEM(metrics, m);
    names[m][0] = PyTuple_GET_ITEM(t, 1);
    names[m][1] = PyTuple_GET_ITEM(t, 2);
    PyObject* hit = PyDict_GET_SIZE(cached) > 0 ? PyDict_GetItemWithError(cached, PyTuple_GET_ITEM(t, 0)) : nullptr;   // borrowed
    if (hit) out[m] = PyFloat_AsDouble(hit);
    else missing |= 1u << m;
    if (PyErr_Occurred()) return -1;
  }
  for (Py_ssize_t i = 0; i < n && missing; ++i) {
    PyObject* rec = PyList_GET_ITEM(records, i);
    if (Py_TYPE(rec) != instance_type) return -1;
    Ref list(field(rec, s__metrics));
    if (!list.p || !PyList_Check(list.p)) return -1;
    for (Py_ssize_t j = 0; j < PyList_GET_SIZE(list.p) && missing; ++j) {
      PyObject* pair = PyList_GET_ITEM(list.p, j);
      if (!PyTuple_Check(pair) || PyTuple_GET_SIZE(pair) != 2) return -1;
      PyObject* key = PyTuple_GET_ITEM(pair, 0);
      int m = 0;
      while (m < 3 && key != names[m][0] && key != names[m][1]) ++m;
      if (m == 3) {
        if (!PyUnicode_Check(key)) return -1;
        for (m = 0; m < 3; ++m)
          if (PyUnicode_Compare(key, names[m][0]) == 0 || PyUnicode_Compare(key, names[m][1]) == 0) break;
      }
      if (m == 3 || !(missing >> m & 1u)) continue;
      out[m] = PyFloat_AsDouble(PyTuple_GET_ITEM(pair, 1));
      if (out[m] == -1.0 && PyErr_Occurred()) return -1;
      missing &= ~(1u << m);
    }
  }
  return missing == 0 ? 1 : 0;
}

// A contiguous buffer (numpy array, bytes) seen as values of T; ok() says whether it holds `count` of them, covers()
// whether at least as many.
template <typename T>
struct Buffer {
  Py_buffer view{};
  bool held = false;
  Buffer(PyObject* o, bool writable) {
    held = PyObject_GetBuffer(o, &view, writable ? PyBUF_WRITABLE | PyBUF_C_CONTIGUOUS : PyBUF_C_CONTIGUOUS) == 0;
    if (!held) PyErr_Clear();
  }
  ~Buffer() { if (held) PyBuffer_Release(&view); }
  Buffer(const Buffer&) = delete;
  Buffer& operator=(const Buffer&) = delete;
  bool covers(int64_t count) const { return held && view.len >= count * static_cast<int64_t>(sizeof(T)); }
  bool ok(int64_t count) const { return held && view.len == count * static_cast<int64_t>(sizeof(T)); }
  T* data() const { return static_cast<T*>(view.buf); }
  int64_t size() const { return held ? view.len / static_cast<int64_t>(sizeof(T)) : 0; }
};

// A Python number as a double; sizes are integers, which PyFloat_AsDouble makes a float object of.
double number(PyObject* o, bool* ok) {
  if (PyLong_CheckExact(o)) {
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(o, &overflow);
    if (!overflow) return static_cast<double>(v);
  }
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) *ok = false;
  return v;
}
// Element i of a tuple or list as a double (borrowed access); *ok is cleared when it is no number.
double item(PyObject* seq, Py_ssize_t i, bool* ok) {
  if (!*ok || (!PyTuple_Check(seq) && !PyList_Check(seq)) || i >= PySequence_Fast_GET_SIZE(seq)) {
    *ok = false;
    return 0.0;
  }
  return number(PySequence_Fast_GET_ITEM(seq, i), ok);
}

constexpr Py_ssize_t kFeatureKinds = 3;   // conv2d, linear, bmm: the kinds with positional extractors
struct Columns {
  Py_ssize_t n = 0;
  long at[8];
};
// The column order of kind `kind` from a tuple of column numbers.
bool columns_of(PyObject* t, long kind, Columns* c) {
  static const Py_ssize_t kColumns[kFeatureKinds] = {8, 4, 4};
  if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) > 8) return false;
  c->n = PyTuple_GET_SIZE(t);
  for (Py_ssize_t i = 0; i < c->n; ++i) {
    c->at[i] = PyLong_AsLong(PyTuple_GET_ITEM(t, i));
    if (c->at[i] < 0 || c->at[i] >= kColumns[kind]) return false;
  }
  return true;
}
// Features of one operation recorded positionally (predictor.py:150-232 of the reference) and its measured ms;
// false when it was recorded otherwise (an error may be set).
bool feature_row(long kind, PyObject* op, PyTypeObject* op_type, PyTypeObject* run_type, const Columns& c, float* row,
                 float* measured) {
  static const Py_ssize_t kArity[kFeatureKinds] = {5, 3, 2};
  if (Py_TYPE(op) != op_type) return false;
  Ref arg(field(op, s__arguments)), f(field(op, s__forward)), b(field(op, s__backward));
  if (!arg.p || !f.p || !b.p || arg.p == Py_None) return false;
  Ref args(get(arg.p, s_args)), kwargs(get(arg.p, s_kwargs));
  if (!args.p || !kwargs.p || !PyTuple_Check(args.p) || !PyDict_Check(kwargs.p) || PyDict_GET_SIZE(kwargs.p) != 0 ||
      PyTuple_GET_SIZE(args.p) < kArity[kind])
    return false;
  PyObject *x = PyTuple_GET_ITEM(args.p, 0), *w = PyTuple_GET_ITEM(args.p, 1);
  bool ok = true;
  double v[8] = {};
  if (kind == 0) {
    auto first = [&](PyObject* o) {
      return PyTuple_Check(o) ? item(o, 0, &ok) : number(o, &ok);
    };
    v[0] = item(x, 0, &ok); v[1] = item(x, 2, &ok); v[2] = item(x, 1, &ok); v[3] = item(w, 0, &ok);
    v[4] = item(w, 2, &ok);
    v[5] = first(PyTuple_GET_ITEM(args.p, 3));
    v[6] = first(PyTuple_GET_ITEM(args.p, 4));
    v[7] = PyTuple_GET_ITEM(args.p, 2) == Py_None ? 0.0 : 1.0;
  } else if (kind == 1) {
    v[0] = 1.0;
    const Py_ssize_t dims = PyTuple_Check(x) || PyList_Check(x) ? PySequence_Fast_GET_SIZE(x) : 0;
    if (dims == 0) return false;
    for (Py_ssize_t d = 0; d + 1 < dims; ++d) v[0] *= item(x, d, &ok);
    v[1] = item(w, 1, &ok);
    v[2] = item(w, 0, &ok);
    v[3] = PyTuple_GET_ITEM(args.p, 2) == Py_None ? 0.0 : 1.0;
  } else {
    v[0] = item(x, 0, &ok); v[1] = item(x, 1, &ok); v[2] = item(x, 2, &ok); v[3] = item(w, 2, &ok);
  }
  double run = 0.0;
  for (PyObject* r : {f.p, b.p}) {
    if (r == Py_None) continue;
    if (Py_TYPE(r) != run_type) return false;
    Ref t(field(r, s__run_time_ms));
    run += t.p ? PyFloat_AsDouble(t.p) : 0.0;
    if (PyErr_Occurred()) return false;
  }
  if (!ok) return false;
  for (Py_ssize_t i = 0; i < c.n; ++i) row[i] = static_cast<float>(v[c.at[i]]);
  *measured = static_cast<float>(run);
  return true;
}

// flatten_trace(operations, (MeasuredOperation, RunTimeMeasurement, MeasuredKernel, KernelInstance),
//               special names, MLP kinds (conv2d, linear, bmm first), metrics ((Metric, name, legacy name) x 3),
//               with_metrics, column orders of the first three kinds, with_names, early or None)
// -> None when the operations are not all of those very classes or not of one device, else
//    (number of kernels, number of passes, names or None, wave_idx, fwd_run, bwd_run, offsets, overheads: bytes of int64 / float64,
//     (indices per MLP kind: bytes of int64), passed-through indices,
//     (num_blocks, block_size, regs, smem, time, gamma), (eff, read, write, has) or None, offsets: CUDA tensors,
//     per kind of the first three: (features, measured ms: CUDA tensors, measured ms as bytes), or None when one of
//     its operations was not recorded positionally, what `early` returned or None, page-locked memory that has to be
//     kept until the stream has got to the end of the upload, or None)
// The operations of the MLP kinds are walked first.  early(the entries per kind of the first three, indices per MLP kind)
// is called when their features are on the GPU, before the walk over the kernels, which takes longer than the
// predictors do: what it launches runs meanwhile.  Where a kind has no features yet (it is not of the first three, or one
// of its operations was not recorded positionally) the features go with the records, and `early` gets None for the entries.
PyObject* flatten_trace(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 9) return not_ordinary();
  Ref ops(PySequence_Tuple(a[0]));   // `early` runs Python, other threads as well: a list may change meanwhile
  if (!ops.p) return nullptr;
  PyTypeObject* type[4];
  for (int i = 0; i < 4; ++i) type[i] = reinterpret_cast<PyTypeObject*>(PyTuple_GET_ITEM(a[1], i));
  PyObject *special = a[2], *kinds = a[3], *metrics = a[4];
  const bool with_metrics = PyObject_IsTrue(a[5]) == 1, with_names = PyObject_IsTrue(a[7]) == 1;
  const Py_ssize_t n = PyTuple_GET_SIZE(ops.p), n_kinds = PyTuple_GET_SIZE(kinds);

  Ref names(with_names ? PyList_New(0) : Py_NewRef(Py_None)), passed(PyList_New(0));
  if (n_kinds < kFeatureKinds || n_kinds > 8) return not_ordinary();
  std::vector<int64_t> kind_idx[8];
  struct Rows {
    Columns c;
    bool ok;
    std::vector<float> f, ms;
  } feats[kFeatureKinds];
  for (long k = 0; k < kFeatureKinds; ++k) feats[k].ok = columns_of(PyTuple_GET_ITEM(a[6], k), k, &feats[k].c);
  std::vector<int64_t> wave_idx, fwd, bwd, offsets{0};
  std::vector<PyObject*> wave_ops;   // borrowed from `ops`
  std::vector<double> overhead, eff, rd, wr;
  std::vector<int32_t> nb;
  std::vector<uint16_t> bs, rg;
  std::vector<uint32_t> sm;
  std::vector<float> tm;
  std::vector<uint8_t> has;
  bool any_metrics = false;
  Ref first_device(nullptr);

  auto add_run = [&](PyObject* run) -> bool {
    if (Py_TYPE(run) != type[1]) return false;
    Ref list(field(run, s__kernels)), ms(field(run, s__run_time_ms));
    if (!list.p || !ms.p || (!PyList_Check(list.p) && !PyTuple_Check(list.p))) return false;
    const double wall = PyFloat_AsDouble(ms.p);
    if (PyErr_Occurred()) return false;
    double busy = 0.0;
    const Py_ssize_t count = PySequence_Fast_GET_SIZE(list.p);
    for (Py_ssize_t i = 0; i < count; ++i) {
      PyObject* k = PySequence_Fast_GET_ITEM(list.p, i);
      if (Py_TYPE(k) != type[2]) return false;
      Ref c(field(k, s__c));
      if (!c.p || Py_TYPE(c.p) != type[3]) return false;
      bool ok = true;
      const int64_t blocks = int_of(c.p, s__num_blocks, &ok), block = int_of(c.p, s__block_size, &ok),
                    regs = int_of(c.p, s__regs, &ok), time = int_of(c.p, s__run_time_ns, &ok),
                    stat = int_of(c.p, s__smem_static, &ok), dyn = int_of(c.p, s__smem_dynamic, &ok);
      if (!ok || blocks != static_cast<int32_t>(blocks)) return false;
      const int64_t smem = stat + dyn;
      nb.push_back(static_cast<int32_t>(blocks));
      bs.push_back(static_cast<uint16_t>(block < 0 ? 0 : (block > 0xFFFF ? 0xFFFF : block)));
      rg.push_back(static_cast<uint16_t>(regs & 0xFFFF));
      sm.push_back(smem >= 0 && smem <= 0xFFFFFFFFll ? static_cast<uint32_t>(smem) : 0xFFFFFFFFu);
      tm.push_back(static_cast<float>(static_cast<double>(time)));
      busy += static_cast<double>(time);
      if (with_names) {
        Ref name(field(c.p, s__name));
        if (!name.p || PyList_Append(names.p, name.p) < 0) return false;
      }
      if (with_metrics) {
        Ref records(field(k, s__metrics_kernels)), cached(field(k, s__cached_metrics));
        if (!records.p || !cached.p || !PyList_Check(records.p) || !PyDict_Check(cached.p)) return false;
        double v[3] = {0.0, 0.0, 0.0};
        const int found = find_metrics(records.p, cached.p, metrics, type[3], v);
        if (found < 0) return false;
        eff.push_back(found ? v[0] : 0.0);
        rd.push_back(found ? v[1] : 0.0);
        wr.push_back(found ? v[2] : 0.0);
        has.push_back(static_cast<uint8_t>(found));
        any_metrics = any_metrics || found;
      }
    }
    offsets.push_back(static_cast<int64_t>(nb.size()));
    // launch overhead of a pass (predictor.py:113-116 of the reference): wall time minus kernel time
    const double rest = wall * 1e6 - busy;
    overhead.push_back(rest > 0.0 ? rest : 0.0);
    return true;
  };

  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* op = PyTuple_GET_ITEM(ops.p, i);
    if (Py_TYPE(op) != type[0]) return not_ordinary();
    Ref name(field(op, s__name)), device(field(op, s__device));
    if (!name.p || !device.p) return not_ordinary();
    if (!first_device.p) {
      first_device.p = Py_NewRef(device.p);
    } else if (device.p != first_device.p) {
      Ref x(get(device.p, s_name)), y(get(first_device.p, s_name));
      if (!x.p || !y.p || PyObject_RichCompareBool(x.p, y.p, Py_EQ) != 1) return not_ordinary();
    }
    const int is_special = PySet_Contains(special, name.p);
    if (is_special < 0) return not_ordinary();
    if (!is_special) {
      wave_idx.push_back(i);
      wave_ops.push_back(op);
      continue;
    }
    Py_ssize_t kind = 0;
    while (kind < n_kinds && PyObject_RichCompareBool(PyTuple_GET_ITEM(kinds, kind), name.p, Py_EQ) != 1) ++kind;
    if (kind == n_kinds) {
      Ref at(PyLong_FromSsize_t(i));
      if (PyList_Append(passed.p, at.p) < 0) return nullptr;
      continue;
    }
    kind_idx[kind].push_back(i);
    if (kind >= kFeatureKinds || !feats[kind].ok) continue;
    Rows& r = feats[kind];
    r.f.resize(r.f.size() + r.c.n);
    r.ms.resize(r.ms.size() + 1);
    r.ok = feature_row(static_cast<long>(kind), op, type[0], type[1], r.c, r.f.data() + r.f.size() - r.c.n,
                       &r.ms.back());
    if (!r.ok) PyErr_Clear();
  }
  if (PyErr_Occurred()) return not_ordinary();

  // what goes to the GPU in one piece, and the tensors in it
  struct Upload {
    struct Piece {
      size_t at;
      int64_t rows, cols;
      at::ScalarType type;
    };
    std::vector<uint8_t> host;
    std::vector<Piece> pieces;
    at::Tensor block;
    size_t taken = 0;
    void put(const void* p, int64_t count, size_t size, at::ScalarType t, int64_t cols = 0) {
      const size_t at0 = (host.size() + 255) & ~static_cast<size_t>(255);
      host.resize(at0 + count * size);
      std::memcpy(host.data() + at0, p, count * size);
      pieces.push_back(Piece{at0, cols ? count / cols : count, cols, t});
    }
    // A copy from pageable memory first waits for what is on the stream; behind `early`'s launches it goes from a
    // page-locked block.
    at::Tensor staged;
    bool go(bool behind) {
      if (host.empty()) return true;
      const int64_t total[1] = {static_cast<int64_t>(host.size())};
      int current = 0;
      cudaGetDevice(&current);
      block = empty(total, at::kByte, at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(current)));
      const void* from = host.data();
      if (behind) {
        staged = at::Tensor(at::detail::empty_cpu(total, at::kByte, /*pin_memory=*/true));
        from = std::memcpy(staged.mutable_data_ptr(), host.data(), host.size());
      }
      const cudaError_t e = cudaMemcpyAsync(block.mutable_data_ptr(), from, host.size(), cudaMemcpyHostToDevice,
                                            static_cast<cudaStream_t>(stream_now()));
      if (e != cudaSuccess) PyErr_Format(PyExc_RuntimeError, "upload of the trace: %s", cudaGetErrorString(e));
      return e == cudaSuccess;
    }
    PyObject* view() {
      const Piece& p = pieces[taken++];
      const int64_t size[2] = {p.rows, p.cols};
      return THPVariable_Wrap(inside(block, p.at, at::IntArrayRef(size, p.cols ? 2 : 1), p.type));
    }
    PyObject* views(Py_ssize_t count) {
      PyObject* t = PyTuple_New(count);
      for (Py_ssize_t i = 0; t && i < count; ++i) PyTuple_SET_ITEM(t, i, view());
      return t;
    }
  };
  Upload records, features;
  Ref special_rows(PyTuple_New(kFeatureKinds)), kinds_out(PyTuple_New(n_kinds)), started(Py_NewRef(Py_None));
  if (!special_rows.p || !kinds_out.p) return nullptr;
  for (Py_ssize_t k = 0; k < n_kinds; ++k) PyTuple_SET_ITEM(kinds_out.p, k, bytes_of(kind_idx[k]));
  // the features go on their own when all kinds can start with them, else with the records
  bool early = a[8] != Py_None, any = false, all = true;
  for (Py_ssize_t k = 0; k < n_kinds; ++k) {
    if (kind_idx[k].empty()) continue;
    any = true;
    all = all && k < kFeatureKinds && feats[k].ok;
  }
  if (early && any && !all) {
    Ref none(PyObject_CallFunctionObjArgs(a[8], Py_None, kinds_out.p, nullptr));
    if (!none.p) return nullptr;
  }
  early = early && any && all;
  Upload& with = early ? features : records;
  auto put_features = [&] {
    for (Rows& r : feats) {
      r.ok = r.ok && !r.ms.empty();
      if (!r.ok) continue;
      with.put(r.f.data(), static_cast<int64_t>(r.f.size()), 4, at::kFloat, r.c.n);
      with.put(r.ms.data(), static_cast<int64_t>(r.ms.size()), 4, at::kFloat);
    }
  };
  auto take_features = [&] {
    for (Py_ssize_t k = 0; k < kFeatureKinds; ++k) {
      PyObject* got = Py_NewRef(Py_None);
      if (feats[k].ok) {
        PyObject *f = with.view(), *m = with.view();
        Py_SETREF(got, Py_BuildValue("(NNN)", f, m, bytes_of(feats[k].ms)));
      }
      PyTuple_SET_ITEM(special_rows.p, k, got);
    }
  };
  if (early) {
    put_features();
    if (!features.go(false)) return nullptr;
    take_features();
    if (PyErr_Occurred()) return nullptr;
    Py_SETREF(started.p, PyObject_CallFunctionObjArgs(a[8], special_rows.p, kinds_out.p, nullptr));
    if (!started.p) return nullptr;
  }

  for (PyObject* op : wave_ops) {
    Ref f(field(op, s__forward)), b(field(op, s__backward));
    if (!f.p || !b.p) return not_ordinary();
    fwd.push_back(static_cast<int64_t>(overhead.size()));
    if (!add_run(f.p)) return not_ordinary();
    bwd.push_back(b.p == Py_None ? -1 : static_cast<int64_t>(overhead.size()));
    if (b.p != Py_None && !add_run(b.p)) return not_ordinary();
  }
  if (PyErr_Occurred()) return not_ordinary();

  const int64_t K = static_cast<int64_t>(nb.size());
  if (K > 0) {
    const std::vector<float> gamma(nb.size(), 1.0f);
    records.put(nb.data(), K, 4, at::kInt);
    records.put(bs.data(), K, 2, at::kUInt16);
    records.put(rg.data(), K, 2, at::kUInt16);
    records.put(sm.data(), K, 4, at::kUInt32);
    records.put(tm.data(), K, 4, at::kFloat);
    records.put(gamma.data(), K, 4, at::kFloat);
    records.put(offsets.data(), static_cast<int64_t>(offsets.size()), 8, at::kLong);
    if (any_metrics) {
      records.put(eff.data(), K, 8, at::kDouble);
      records.put(rd.data(), K, 8, at::kDouble);
      records.put(wr.data(), K, 8, at::kDouble);
      records.put(has.data(), K, 1, at::kByte);
    }
  }
  if (!early) put_features();
  if (!records.go(started.p != Py_None)) return nullptr;
  Ref soa(Py_NewRef(Py_None)), met(Py_NewRef(Py_None)), off(Py_NewRef(Py_None));
  if (K > 0) {
    Py_SETREF(soa.p, records.views(6));
    Py_SETREF(off.p, records.view());
    if (any_metrics) Py_SETREF(met.p, records.views(4));
  }
  if (!early) take_features();
  if (PyErr_Occurred() || !soa.p || !off.p || !met.p) return nullptr;
  Ref staged(records.staged.defined() ? THPVariable_Wrap(records.staged) : Py_NewRef(Py_None));
  if (!staged.p) return nullptr;
  return Py_BuildValue("(LLONNNNNOOOOOOOO)", static_cast<long long>(K), static_cast<long long>(overhead.size()), names.p, bytes_of(wave_idx), bytes_of(fwd), bytes_of(bwd),
                       bytes_of(offsets), bytes_of(overhead), kinds_out.p, passed.p, soa.p, met.p, off.p, special_rows.p, started.p, staged.p);
  END_HANDLE_TH_ERRORS
}

// submit_wave(block, device block, kernels, origin, dests, out, partials or None, totals or None,
//             [(host tensor, device tensor)], (upload, compute, download stream handles),
//             (uploaded, computed, downloaded event handles), used)
// One batch of hostio.WaveScaleHost: upload of a record block, wave scaling, download of the wanted results on
// three streams that events tie together.  `used`: the slot's buffers have held a batch before.
PyObject* submit_wave(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 12 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !PyList_Check(a[8]) || !PyTuple_Check(a[9]) ||
      !PyTuple_Check(a[10])) {
    PyErr_SetString(PyExc_TypeError, "submit_wave: bad arguments");
    return nullptr;
  }
  cudaStream_t s[3];
  cudaEvent_t ev[3];
  for (int i = 0; i < 3; ++i) {
    s[i] = static_cast<cudaStream_t>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(a[9], i)));
    ev[i] = static_cast<cudaEvent_t>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(a[10], i)));
  }
  const bool used = PyObject_IsTrue(a[11]) == 1;
  if (PyErr_Occurred()) return nullptr;
  auto ok = [](cudaError_t e) {
    if (e == cudaSuccess) return true;
    PyErr_Format(PyExc_RuntimeError, "submit_wave: %s", cudaGetErrorString(e));
    return false;
  };
  // a page-locked tensor that its owner drops is not reused before the stream has come this far
  auto copy = [&](const at::Tensor& dst, const at::Tensor& src, cudaStream_t stream) {
    if (!ok(cudaMemcpyAsync(dst.mutable_data_ptr(), src.data_ptr(), dst.nbytes(), cudaMemcpyDefault, stream))) return false;
    const at::Tensor& host = src.is_cuda() ? dst : src;
    const at::Device dev = (src.is_cuda() ? src : dst).device();
    if (!host.is_cuda())
      at::getHostAllocator(at::kCUDA)->record_event(host.mutable_data_ptr(), host.storage().data_ptr().get_context(),
                                                    c10::cuda::getStreamFromExternal(stream, dev.index()).unwrap());
    return true;
  };
  const at::Tensor &block = THPVariable_Unpack(a[0]), &dev_block = THPVariable_Unpack(a[1]);
  const c10::DeviceIndex index = dev_block.device().index();
  // the slot's device inputs were last read by the kernel of batch (i - depth)
  if (used && !ok(cudaStreamWaitEvent(s[0], ev[1], 0))) return nullptr;
  if (!copy(dev_block, block, s[0]) || !ok(cudaEventRecord(ev[0], s[0])) || !ok(cudaStreamWaitEvent(s[1], ev[0], 0)))
    return nullptr;
  // the kernel of this batch overwrites outputs the download of batch (i - depth) reads
  if (used && !ok(cudaStreamWaitEvent(s[1], ev[2], 0))) return nullptr;
  {
    c10::cuda::CUDAStreamGuard guard(c10::cuda::getStreamFromExternal(s[1], index));
    PyObject* args[9] = {a[2], a[3], a[4], Py_None, Py_None, Py_False, Py_False, a[5], a[6]};
    Ref r(wave_scale(nullptr, args, 9));
    if (!r.p) return nullptr;
    if (r.p == Py_None) Py_RETURN_NONE;
    if (a[6] != Py_None) {
      Ref buffer(PyObject_GetAttr(a[6], s_buffer)), per(PyObject_GetAttr(a[6], s_per_plane)),
          planes(PyObject_GetAttr(a[6], s_n_planes));
      if (!buffer.p || !per.p || !planes.p) return nullptr;
      PyObject* sum[4] = {buffer.p, per.p, planes.p, a[7]};
      Ref t(partials_sum(nullptr, sum, 4));
      if (!t.p) return nullptr;
      if (t.p == Py_None) Py_RETURN_NONE;
    }
  }
  if (!ok(cudaEventRecord(ev[1], s[1])) || !ok(cudaStreamWaitEvent(s[2], ev[1], 0))) return nullptr;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[8]); ++i) {
    PyObject* t = PyList_GET_ITEM(a[8], i);
    if (!copy(THPVariable_Unpack(PyTuple_GET_ITEM(t, 0)), THPVariable_Unpack(PyTuple_GET_ITEM(t, 1)), s[2])) return nullptr;
  }
  if (!ok(cudaEventRecord(ev[2], s[2]))) return nullptr;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------
// Page-locked memory for host results
// ---------------------------------------------------------------------------
// Arrays over such blocks are what batched.wave_scale_host returns: the kernel writes them directly.  A block
// goes back to the pool when the last array over it goes.  Blocks come in quarter steps between powers of two,
// of at most kMostBlock bytes and kMostTotal in all, room for a few results of a million kernels on eight devices;
// a caller who keeps more results than that gets the rest in ordinary memory, as does one who asks for a
// larger block.
//
// Page-locking costs about 0.3 ms per MB, so it must not recur: 65,536 kernels on six devices take 0.16 ms into a
// block that has come back, 1.0 ms into fresh pages and 2.2 ms with a new block.  So a new one needs credit: two to
// begin with (a loop that keeps one result while the next is made), one more for each time a block is used again,
// kMostCredit at most.  A caller who keeps every result pays for two blocks and then gets ordinary memory; so does
// one whose sizes push one another out of the pool.
constexpr size_t kMostBlock = 128 << 20, kMostTotal = 256 << 20;
constexpr int kFirstCredit = 2, kMostCredit = 8;
struct HostBlocks {
  std::mutex mu;
  std::vector<std::pair<size_t, void*>> idle;
  size_t total = 0, blocks = 0;
  int credit = kFirstCredit;
};
HostBlocks& host_blocks() {
  static HostBlocks* b = new HostBlocks();   // never destroyed: arrays may outlive the interpreter's own clean-up
  return *b;
}
struct HostBlock {
  PyObject_HEAD
  void* ptr;
  size_t bytes;      // of the block
  Py_ssize_t asked;
};
void host_block_dealloc(PyObject* o) {
  HostBlock* b = reinterpret_cast<HostBlock*>(o);
  if (b->ptr) {
    HostBlocks& pool = host_blocks();
    std::lock_guard<std::mutex> lock(pool.mu);
    pool.idle.emplace_back(b->bytes, b->ptr);
  }
  Py_TYPE(o)->tp_free(o);
}
int host_block_buffer(PyObject* o, Py_buffer* view, int flags) {
  HostBlock* b = reinterpret_cast<HostBlock*>(o);
  return PyBuffer_FillInfo(view, o, b->ptr, b->asked, 0, flags);
}
PyBufferProcs host_block_procs = {host_block_buffer, nullptr};
PyTypeObject host_block_type = [] {
  PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name = "habitat_b200._binding.HostBlock";
  t.tp_basicsize = sizeof(HostBlock);
  t.tp_flags = Py_TPFLAGS_DEFAULT;
  t.tp_dealloc = host_block_dealloc;
  t.tp_as_buffer = &host_block_procs;
  return t;
}();

// host_block(bytes) -> an object with a writable buffer in page-locked memory, or None (see above)
PyObject* host_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 1) Py_RETURN_NONE;
  const Py_ssize_t asked = PyLong_AsSsize_t(a[0]);
  if (PyErr_Occurred()) return nullptr;
  if (asked < 0 || static_cast<size_t>(asked) > kMostBlock) Py_RETURN_NONE;
  size_t top = 4096;
  while (top < static_cast<size_t>(asked)) top *= 2;
  size_t bytes = top / 2;
  while (bytes < static_cast<size_t>(asked) || bytes < 4096) bytes += top / 8;
  HostBlocks& pool = host_blocks();
  void* ptr = nullptr;
  {
    std::lock_guard<std::mutex> lock(pool.mu);
    // the smallest idle block that is large enough, and not more than twice as large
    auto best = pool.idle.end();
    for (auto it = pool.idle.begin(); it != pool.idle.end(); ++it)
      if (it->first >= bytes && it->first <= 2 * bytes && (best == pool.idle.end() || it->first < best->first)) best = it;
    if (best != pool.idle.end()) {
      bytes = best->first;
      ptr = best->second;
      pool.idle.erase(best);
      if (pool.credit < kMostCredit) ++pool.credit;
    } else if (pool.credit > 0) {
      // make room by giving back idle blocks of other sizes
      while (pool.total + bytes > kMostTotal && !pool.idle.empty()) {
        pool.total -= pool.idle.back().first;
        --pool.blocks;
        cudaFreeHost(pool.idle.back().second);
        pool.idle.pop_back();
      }
      try {
        pool.idle.reserve(pool.blocks + 1);   // a block that comes back needs no memory
      } catch (const std::bad_alloc&) {
        Py_RETURN_NONE;
      }
      if (pool.total + bytes <= kMostTotal) {
        if (cudaHostAlloc(&ptr, bytes, cudaHostAllocPortable) == cudaSuccess) {
          pool.total += bytes;
          ++pool.blocks;
          --pool.credit;
        } else {
          cudaGetLastError();
          ptr = nullptr;
        }
      }
    }
  }
  if (!ptr) Py_RETURN_NONE;
  HostBlock* b = PyObject_New(HostBlock, &host_block_type);
  if (!b) {
    std::lock_guard<std::mutex> lock(pool.mu);
    pool.idle.emplace_back(bytes, ptr);
    return nullptr;
  }
  b->ptr = ptr;
  b->bytes = bytes;
  b->asked = asked;
  return reinterpret_cast<PyObject*>(b);
}
// release_host_blocks(): gives the idle blocks back
PyObject* release_host_blocks(PyObject*, PyObject* const*, Py_ssize_t) {
  HostBlocks& pool = host_blocks();
  std::lock_guard<std::mutex> lock(pool.mu);
  for (auto& b : pool.idle) {
    cudaFreeHost(b.second);
    pool.total -= b.first;
    --pool.blocks;
  }
  pool.idle.clear();
  Py_RETURN_NONE;
}

// wave_scale_host(num_blocks, block_size, regs, smem, time, gamma, origin, dests,
//                 (scaled, occupancy, waves, origin occupancy, origin waves, status or None, limits or None))
// -> True, or None when a buffer does not fit
PyObject* wave_scale_host(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 9 || !PyTuple_Check(a[8]) || PyTuple_GET_SIZE(a[8]) != 7) Py_RETURN_NONE;
  Ref dests(PySequence_Fast(a[7], "dests must be a sequence of DeviceProperties"));
  if (!dests.p) return nullptr;
  const Py_ssize_t D = PySequence_Fast_GET_SIZE(dests.p);
  if (D > HB_MAX_DEVICES) Py_RETURN_NONE;
  const Buffer<int32_t> nb(a[0], false);
  const Buffer<uint16_t> bs(a[1], false), rg(a[2], false);
  const Buffer<uint32_t> sm(a[3], false);
  const Buffer<float> tm(a[4], false), gm(a[5], false);
  const int64_t K = nb.size();
  if (!nb.held || !bs.covers(K) || !rg.covers(K) || !sm.covers(K) || !tm.covers(K) || !gm.covers(K)) Py_RETURN_NONE;
  const long origin = row_of(a[6]);
  if (origin < 0) return nullptr;
  int32_t rows[HB_MAX_DEVICES];
  for (Py_ssize_t d = 0; d < D; ++d) {
    const long r = row_of(PySequence_Fast_GET_ITEM(dests.p, d));
    if (r < 0) return nullptr;
    rows[d] = static_cast<int32_t>(r);
  }
  auto result = [&](int i) { return PyTuple_GET_ITEM(a[8], i); };
  const Buffer<float> ns(result(0), true);
  const Buffer<uint8_t> occ(result(1), true), oocc(result(3), true);
  const Buffer<uint32_t> wav(result(2), true), owav(result(4), true);
  if (!ns.ok(D * K) || !occ.ok(D * K) || !wav.ok(D * K) || !oocc.ok(K) || !owav.ok(K)) Py_RETURN_NONE;
  hb_wave_out out{ns.data(), occ.data(), wav.data(), oocc.data(), owav.data(), nullptr, nullptr};
  const Buffer<uint8_t> status(result(5), true);
  const Buffer<int32_t> limits(result(6), true);
  if (result(5) != Py_None) {
    if (!status.ok(D * K)) Py_RETURN_NONE;
    out.status = status.data();
  }
  if (result(6) != Py_None) {
    if (!limits.ok((D + 1) * 4 * K)) Py_RETURN_NONE;
    out.limits = limits.data();
  }
  const hb_kernel_soa k{nb.data(), bs.data(), rg.data(), sm.data(), tm.data(), gm.data()};
  hb_status st;
  Py_BEGIN_ALLOW_THREADS
  st = api.wave_scale_host(&k, K, static_cast<int32_t>(origin), rows, static_cast<int32_t>(D), nullptr, &out);
  Py_END_ALLOW_THREADS
  if (failed(st)) return nullptr;
  Py_RETURN_TRUE;
}

// The operations of one MLP kind of a trace: the predictor, its inputs, and where its raw predictions (device) and
// the operations' times (page-locked) go.
struct Kind {
  hb_mlp* h;
  const at::Tensor *f, *ms;
  const uint8_t* rows;
  const int64_t* idx;
  int64_t n;
  float *pred, *times;
};
size_t place(size_t* at, size_t bytes) {
  const size_t here = *at;
  *at = (here + bytes + 255) & ~static_cast<size_t>(255);
  return here;
}
// Kinds of a list of (handle address, features, measured ms, device rows (bytes: origin, then T destinations), operation
// indices (int64, below n_ops)), without their places; null or what is wrong with it.
const char* kinds_of(PyObject* list, int64_t T, int64_t n_ops, std::vector<Kind>* kinds) {
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
    PyObject* t = PyList_GET_ITEM(list, i);
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 5) return "operation kind";
    Kind k{};
    k.h = static_cast<hb_mlp*>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(t, 0)));
    k.f = tensor(PyTuple_GET_ITEM(t, 1), at::kFloat);
    k.ms = tensor(PyTuple_GET_ITEM(t, 2), at::kFloat);
    PyObject* rows = PyTuple_GET_ITEM(t, 3);
    const Buffer<int64_t> idx(PyTuple_GET_ITEM(t, 4), false);   // the tuple keeps the memory alive
    if (!k.f || k.f->dim() != 2 || !k.ms || !PyBytes_Check(rows) || PyBytes_GET_SIZE(rows) != T + 1 ||
        k.ms->numel() != k.f->size(0) || !idx.ok(k.f->size(0)))
      return "operation kind";
    k.rows = reinterpret_cast<const uint8_t*>(PyBytes_AS_STRING(rows));
    k.idx = idx.data();
    k.n = k.f->size(0);
    for (int64_t j = 0; j < k.n; ++j)
      if (k.idx[j] < 0 || k.idx[j] >= n_ops) return "operation index";
    kinds->push_back(k);
  }
  return nullptr;
}
bool launch_kinds(const std::vector<Kind>& kinds, int64_t T, cudaStream_t s) {
  std::vector<hb_mlp_grid> grids;
  std::vector<hb_scale_grid> scales;
  for (const Kind& k : kinds) {
    grids.push_back(hb_mlp_grid{k.h, static_cast<const float*>(data(k.f)), k.n, k.rows, static_cast<int32_t>(T + 1), k.pred});
    scales.push_back(hb_scale_grid{static_cast<const float*>(data(k.ms)), k.pred, k.n, static_cast<int32_t>(T), k.times, nullptr});
  }
  return !failed(api.mlp_predict_grid(grids.data(), static_cast<int32_t>(grids.size()), s)) &&
         !failed(api.special_scale_grid(scales.data(), static_cast<int32_t>(scales.size()), s));
}
size_t pred_bytes(const Kind& k, int64_t T) { return static_cast<size_t>(T + 1) * k.n * 4; }
size_t times_bytes(const Kind& k, int64_t T) { return static_cast<size_t>(T) * k.n * 4; }

// Predictors that were started ahead of the rest of a trace: start_kinds makes one, run_group takes its results.  Whoever
// lets go of it waits for what has been launched, which writes to its memory.
constexpr const char* kStartedName = "habitat_b200.started";
struct Started {
  at::Tensor block, host;
  cudaStream_t s = nullptr;
  int64_t T = 0;
  Ref held{nullptr};          // the predictors, and what `kinds` points into
  std::vector<Kind> kinds;
  bool launched = false;
  ~Started() {
    if (launched) cudaStreamSynchronize(s);
  }
};
// start_kinds([as for run_group], destinations, operations, objects that keep the handles alive) -> capsule
PyObject* start_kinds(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 4 || !PyList_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "start_kinds: bad arguments");
    return nullptr;
  }
  std::unique_ptr<Started> st(new Started);
  st->T = PyLong_AsLongLong(a[1]);
  const int64_t n_ops = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (const char* wrong = kinds_of(a[0], st->T, n_ops, &st->kinds)) {
    PyErr_Format(PyExc_TypeError, "start_kinds: %s", wrong);
    return nullptr;
  }
  Ref list(PySequence_Tuple(a[0])), handles(PySequence_Tuple(a[3]));
  if (!list.p || !handles.p) return nullptr;
  st->held.p = PyTuple_Pack(2, list.p, handles.p);
  if (!st->held.p) return nullptr;
  size_t pinned = 0, device = 0;
  std::vector<std::pair<size_t, size_t>> at;
  for (const Kind& k : st->kinds) at.emplace_back(place(&device, pred_bytes(k, st->T)), place(&pinned, times_bytes(k, st->T)));
  int current = 0;
  cudaGetDevice(&current);
  const int64_t dev_size[1] = {static_cast<int64_t>(device ? device : 16)},
                host_size[1] = {static_cast<int64_t>(pinned ? pinned : 16)};
  st->block = empty(dev_size, at::kByte, at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(current)));
  st->host = at::Tensor(at::detail::empty_cpu(host_size, at::kByte, /*pin_memory=*/true));
  for (size_t i = 0; i < st->kinds.size(); ++i) {
    st->kinds[i].pred = reinterpret_cast<float*>(static_cast<uint8_t*>(st->block.mutable_data_ptr()) + at[i].first);
    st->kinds[i].times = reinterpret_cast<float*>(static_cast<uint8_t*>(st->host.mutable_data_ptr()) + at[i].second);
  }
  st->s = static_cast<cudaStream_t>(stream_now());
  st->launched = true;
  if (!launch_kinds(st->kinds, st->T, st->s)) return nullptr;
  PyObject* capsule = PyCapsule_New(st.get(), kStartedName, [](PyObject* c) {
    delete static_cast<Started*>(PyCapsule_GetPointer(c, kStartedName));
  });
  if (capsule) st.release();
  return capsule;
  END_HANDLE_TH_ERRORS
}

// run_group(kernels or None, metrics or None, origin, dests, dest_regs or None, offsets or None,
//           [(handle address, features, measured ms, device rows (bytes: origin, then the destinations),
//             operation indices (int64))],
//           (overheads, wave_idx, fwd_run, bwd_run: float64 / int64), times [T][K] float32,
//           totals [T][passes] float64, ms [T][n] float64 [, what start_kinds returned for these kinds])
// -> (NaN seen, total ms per destination, [per kind: None, or [1 + T][n] float32 predictions as bytes when one
//    may have been clamped]).  One prediction of a flattened trace: fills `times` and `totals` (the kernels' times
// and their sums per pass) and the entries of `ms` of the wave-scaled and MLP-predicted operations; the other
// entries of `ms` are the caller's and are part of the totals.
//
// Two groups of launches: wave scaling with the sums of its passes, and the MLPs of all kinds side by side with
// their ratios.  Both leave their results in page-locked memory themselves.  With many kernels the wave scaling
// goes first, and its results are sorted into the operations while the predictors run; with few it goes last,
// so that the predictors, which take longest, start first.
PyObject* run_group(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if ((n_args != 11 && n_args != 12) || !PyList_Check(a[6]) || !PyTuple_Check(a[7]) || PyTuple_GET_SIZE(a[7]) != 4) {
    PyErr_SetString(PyExc_TypeError, "run_group: bad arguments");
    return nullptr;
  }
  auto refuse = [](const char* what) -> PyObject* {
    PyErr_Format(PyExc_TypeError, "run_group: %s", what);
    return nullptr;
  };
  Ref dests(PySequence_Fast(a[3], "dests must be a sequence of DeviceProperties"));
  if (!dests.p) return nullptr;
  const int64_t T = PySequence_Fast_GET_SIZE(dests.p);
  if (T > HB_MAX_DEVICES) return refuse("too many destinations");
  const bool scale = a[0] != Py_None;
  int64_t K = 0, n_runs = 0;
  const at::Tensor* off = nullptr;
  if (scale) {
    const Field nb(a[0], s_num_blocks, at::kInt);
    off = tensor(a[5], at::kLong);
    if (!nb.t || !off || off->numel() < 1) return refuse("kernels");
    K = nb.t->numel();
    n_runs = off->numel() - 1;
  }
  const Buffer<double> overhead(PyTuple_GET_ITEM(a[7], 0), false), totals(a[9], true), ms(a[10], true);
  const Buffer<int64_t> wave_idx(PyTuple_GET_ITEM(a[7], 1), false), fwd(PyTuple_GET_ITEM(a[7], 2), false),
      bwd(PyTuple_GET_ITEM(a[7], 3), false);
  const Buffer<float> times(a[8], true);
  const int64_t n_wave = wave_idx.size(), n_ops = T ? ms.size() / T : 0;
  if (scale && (!times.ok(T * K) || !totals.ok(T * n_runs) || !overhead.ok(n_runs))) return refuse("results");
  if (!ms.ok(T * n_ops) || !fwd.ok(n_wave) || !bwd.ok(n_wave)) return refuse("operations");
  if (scale)
    for (int64_t i = 0; i < n_wave; ++i)
      if (wave_idx.data()[i] < 0 || wave_idx.data()[i] >= n_ops || fwd.data()[i] < 0 || fwd.data()[i] >= n_runs ||
          bwd.data()[i] >= n_runs)
        return refuse("operations");

  // in page-locked memory: sums and times of the wave scaling, ms per kind
  size_t pinned = 0, device = 0;
  const size_t h_totals = place(&pinned, static_cast<size_t>(T) * n_runs * 8);
  const size_t h_times = place(&pinned, static_cast<size_t>(T) * K * 4);
  std::vector<Kind> kinds;
  if (const char* wrong = kinds_of(a[6], T, n_ops, &kinds)) return refuse(wrong);
  Started* started = nullptr;
  if (n_args == 12) {
    started = static_cast<Started*>(PyCapsule_GetPointer(a[11], kStartedName));
    if (!started) return nullptr;
    bool same = started->T == T && started->kinds.size() == kinds.size();
    for (size_t i = 0; same && i < kinds.size(); ++i)
      same = kinds[i].h == started->kinds[i].h && kinds[i].n == started->kinds[i].n && kinds[i].f == started->kinds[i].f &&
             kinds[i].ms == started->kinds[i].ms && std::memcmp(kinds[i].rows, started->kinds[i].rows, T + 1) == 0;
    if (!same) return refuse("other kinds than were started");
  }
  std::vector<std::pair<size_t, size_t>> at;
  if (!started)
    for (const Kind& k : kinds) at.emplace_back(place(&device, pred_bytes(k, T)), place(&pinned, times_bytes(k, T)));
  const size_t pairs = static_cast<size_t>(T) * K;
  const size_t d_scaled = place(&device, pairs * 4), d_occ = place(&device, pairs), d_waves = place(&device, pairs * 4),
               d_oocc = place(&device, K), d_owaves = place(&device, static_cast<size_t>(K) * 4);

  int current = 0;
  cudaGetDevice(&current);
  const int64_t dev_size[1] = {static_cast<int64_t>(device ? device : 16)},
                host_size[1] = {static_cast<int64_t>(pinned ? pinned : 16)};
  at::Tensor block = empty(dev_size, at::kByte, at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(current)));
  at::Tensor host(at::detail::empty_cpu(host_size, at::kByte, /*pin_memory=*/true));
  uint8_t* d = static_cast<uint8_t*>(block.mutable_data_ptr());
  uint8_t* h = static_cast<uint8_t*>(host.mutable_data_ptr());
  cudaStream_t s = static_cast<cudaStream_t>(stream_now());
  // whatever has been launched writes to `host`: nobody leaves before it has ended
  struct Settle {
    cudaStream_t s;
    bool on = true;
    ~Settle() { if (on) cudaStreamSynchronize(s); }
  } settle{s};

  for (size_t i = 0; i < kinds.size(); ++i) {
    kinds[i].pred = started ? started->kinds[i].pred : reinterpret_cast<float*>(d + at[i].first);
    kinds[i].times = started ? started->kinds[i].times : reinterpret_cast<float*>(h + at[i].second);
  }
  auto launch_mlps = [&]() -> bool { return started || launch_kinds(kinds, T, s); };
  auto launch_waves = [&]() -> bool {
    if (!scale || K == 0) return true;
    const Field nb(a[0], s_num_blocks, at::kInt), bs(a[0], s_block_size, at::kUInt16), rg(a[0], s_regs, at::kUInt16),
        sm(a[0], s_smem, at::kUInt32), tm(a[0], s_time, at::kFloat), gm(a[0], s_gamma, at::kFloat);
    const at::Tensor* dr = a[4] == Py_None ? nullptr : tensor(a[4], at::kShort);
    if (!bs.covers(K) || !rg.covers(K) || !sm.covers(K) || !tm.covers(K) || !gm.covers(K) ||
        (a[4] != Py_None && (!dr || dr->numel() != T * K)))
      return refuse("kernel records") != nullptr;
    int32_t rows[HB_MAX_DEVICES];
    const long origin = row_of(a[2]);
    if (origin < 0) return false;
    for (int64_t t = 0; t < T; ++t) {
      const long r = row_of(PySequence_Fast_GET_ITEM(dests.p, t));
      if (r < 0) return false;
      rows[t] = static_cast<int32_t>(r);
    }
    const hb_kernel_soa soa{static_cast<const int32_t*>(nb.ptr()), static_cast<const uint16_t*>(bs.ptr()),
                            static_cast<const uint16_t*>(rg.ptr()), static_cast<const uint32_t*>(sm.ptr()),
                            static_cast<const float*>(tm.ptr()), static_cast<const float*>(gm.ptr())};
    const hb_wave_out o{reinterpret_cast<float*>(d + d_scaled), d + d_occ, reinterpret_cast<uint32_t*>(d + d_waves),
                        d + d_oocc, reinterpret_cast<uint32_t*>(d + d_owaves), nullptr, nullptr};
    hb_kernel_metrics m{};
    if (a[1] != Py_None) {
      const Field fe(a[1], s_flop, at::kDouble), rd(a[1], s_rd, at::kDouble), wr(a[1], s_wr, at::kDouble),
          has(a[1], s_has, at::kByte);
      if (!fe.covers(K) || !rd.covers(K) || !wr.covers(K) || !has.covers(K)) return refuse("metrics") != nullptr;
      m = hb_kernel_metrics{static_cast<const double*>(fe.ptr()), static_cast<const double*>(rd.ptr()),
                            static_cast<const double*>(wr.ptr()), static_cast<const uint8_t*>(has.ptr())};
    }
    return !failed(wave_scale_call(soa, a[1] != Py_None ? &m : nullptr, K, static_cast<int32_t>(origin), rows,
                                   static_cast<int32_t>(T), static_cast<const int16_t*>(data(dr)), o, nullptr, nullptr, s)) &&
           !failed(api.segment_sum_planes(o.scaled_ns, K, static_cast<int32_t>(T), static_cast<const int64_t*>(data(off)),
                                          n_runs, reinterpret_cast<double*>(h + h_totals),
                                          reinterpret_cast<float*>(h + h_times), s));
  };
  bool nan = false;
  auto sort_passes = [&] {
    if (!scale) return;
    const double* tot = reinterpret_cast<const double*>(h + h_totals);
    if (K == 0) std::memset(h + h_totals, 0, static_cast<size_t>(T) * n_runs * 8);
    std::memcpy(totals.data(), tot, static_cast<size_t>(T) * n_runs * 8);
    std::memcpy(times.data(), h + h_times, pairs * 4);
    // a NaN time makes its pass's sum NaN, and every kernel is of a pass
    const double* over = overhead.data();
    const int64_t *wi = wave_idx.data(), *fw = fwd.data(), *bw = bwd.data();
    for (int64_t t = 0; t < T; ++t) {
      const double* q = totals.data() + t * n_runs;
      for (int64_t r = 0; r < n_runs; ++r) nan = nan || q[r] != q[r];
      double* out = ms.data() + t * n_ops;
      for (int64_t i = 0; i < n_wave; ++i) {
        double v = (over[fw[i]] + q[fw[i]]) / 1e6;
        if (bw[i] >= 0) v += (over[bw[i]] + q[bw[i]]) / 1e6;
        out[wi[i]] = v;
      }
    }
  };
  std::vector<double> sum_ms(static_cast<size_t>(T), 0.0);
  auto sort_waves = [&] {
    sort_passes();
    // the rows' sums but for the predictors' operations, whose times come later
    for (int64_t t = 0; t < T; ++t) {
      double sum[4] = {0.0, 0.0, 0.0, 0.0};
      double* row = ms.data() + t * n_ops;
      for (const Kind& k : kinds)
        for (int64_t j = 0; j < k.n; ++j) row[k.idx[j]] = 0.0;
      for (int64_t i = 0; i < n_ops; ++i) sum[i & 3] += row[i];
      sum_ms[t] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
  };

  constexpr int64_t kManyPairs = 16384;
  cudaError_t e = cudaSuccess;
  if (scale && !kinds.empty() && !started && T * K >= kManyPairs) {
    struct Event {
      cudaEvent_t ev = nullptr;
      ~Event() { if (ev) cudaEventDestroy(ev); }
    } done;
    e = cudaEventCreateWithFlags(&done.ev, cudaEventDisableTiming);
    if (!launch_waves()) return nullptr;
    if (e == cudaSuccess) e = cudaEventRecord(done.ev, s);
    if (!launch_mlps()) return nullptr;
    Py_BEGIN_ALLOW_THREADS
    if (e == cudaSuccess) e = cudaEventSynchronize(done.ev);
    if (e == cudaSuccess) sort_waves();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    Py_END_ALLOW_THREADS
  } else {
    if (!launch_mlps() || !launch_waves()) return nullptr;
    Py_BEGIN_ALLOW_THREADS
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && started && started->s != s) e = cudaStreamSynchronize(started->s);
    if (e == cudaSuccess) sort_waves();
    Py_END_ALLOW_THREADS
  }
  settle.on = false;
  if (started && e == cudaSuccess) started->launched = false;   // ended
  if (e != cudaSuccess) {
    PyErr_Format(PyExc_RuntimeError, "prediction of a trace: %s", cudaGetErrorString(e));
    return nullptr;
  }
  Ref clamped(PyList_New(static_cast<Py_ssize_t>(kinds.size())));
  for (size_t i = 0; i < kinds.size(); ++i) {
    const Kind& k = kinds[i];
    int32_t code = 0;
    if (failed(api.mlp_poll_status(k.h, &code))) return nullptr;
    const float* v = k.times;
    bool zero = false;
    for (int64_t t = 0; t < T; ++t) {
      double* out = ms.data() + t * n_ops;
      double sum[4] = {0.0, 0.0, 0.0, 0.0};
      for (int64_t j = 0; j < k.n; ++j) {
        const double x = static_cast<double>(v[t * k.n + j]);
        zero = zero || x == 0.0;
        out[k.idx[j]] = x;
        sum[j & 3] += x;
      }
      sum_ms[t] += (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
    PyObject* pred = Py_NewRef(Py_None);
    if (zero) {
      // rare: the raw predictions, for the caller's warnings
      const size_t bytes = pred_bytes(k, T);
      Py_DECREF(pred);
      pred = PyBytes_FromStringAndSize(nullptr, static_cast<Py_ssize_t>(bytes));
      if (!pred) return nullptr;
      if (cudaMemcpy(PyBytes_AS_STRING(pred), k.pred, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) {
        Py_DECREF(pred);
        PyErr_SetString(PyExc_RuntimeError, "run_group: cudaMemcpy");
        return nullptr;
      }
    }
    PyList_SET_ITEM(clamped.p, static_cast<Py_ssize_t>(i), pred);
  }
  Ref sums(PyList_New(static_cast<Py_ssize_t>(T)));
  for (int64_t t = 0; t < T; ++t) {
    PyList_SET_ITEM(sums.p, static_cast<Py_ssize_t>(t), PyFloat_FromDouble(sum_ms[t]));
  }
  return Py_BuildValue("(NOO)", PyBool_FromLong(nan), sums.p, clamped.p);
  END_HANDLE_TH_ERRORS
}

// iteration_totals(kernels, scaled_ns, overhead_ns, kernel_offsets, same (bytes per destination),
//                  [(handle address, features, measured ms, offsets, device rows (bytes))])
// -> [I, D] float64 totals (habitat_b200/iteration.py), or None when an argument does not fit
PyObject* iteration_totals(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 6 || !PyBytes_Check(a[4]) || !PyList_Check(a[5])) return not_ordinary();
  const Field tm(a[0], s_time, at::kFloat);
  const at::Tensor *scaled = tensor(a[1], at::kFloat), *over = tensor(a[2], at::kFloat), *off = tensor(a[3], at::kLong);
  if (!tm.t || !scaled || !over || !off || off->numel() < 1) return not_ordinary();
  const int64_t K = tm.t->numel(), I = off->numel() - 1, D = PyBytes_GET_SIZE(a[4]);
  if (over->numel() < K || scaled->numel() != D * K) return not_ordinary();
  const uint8_t* same = reinterpret_cast<const uint8_t*>(PyBytes_AS_STRING(a[4]));
  int64_t others = 0;   // destinations that the kinds are predicted for
  for (int64_t d = 0; d < D; ++d) others += same[d] == 0;
  struct Kind { hb_mlp* h; const at::Tensor *f, *ms, *off; const uint8_t* rows; int64_t blocks; };
  std::vector<Kind> kinds;
  int64_t floats = 0;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[5]); ++i) {
    PyObject* t = PyList_GET_ITEM(a[5], i);
    Kind k{static_cast<hb_mlp*>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(t, 0))), tensor(PyTuple_GET_ITEM(t, 1), at::kFloat),
           tensor(PyTuple_GET_ITEM(t, 2), at::kFloat), tensor(PyTuple_GET_ITEM(t, 3), at::kLong),
           reinterpret_cast<const uint8_t*>(PyBytes_AS_STRING(PyTuple_GET_ITEM(t, 4))),
           PyBytes_GET_SIZE(PyTuple_GET_ITEM(t, 4))};
    if (!k.f || !k.ms || !k.off || k.f->dim() != 2 || k.ms->numel() != k.f->size(0) || k.off->numel() != I + 1 ||
        k.blocks != 1 + others)
      return not_ordinary();
    kinds.push_back(k);
    if (k.blocks > 1) floats += (k.blocks * k.f->size(0) + 63) & ~int64_t{63};
  }
  const int64_t id[2] = {I, D}, fl[1] = {floats};
  at::Tensor out = empty(id, at::kDouble, tm.t->device()), preds = empty(fl, at::kFloat, tm.t->device());
  float* p = static_cast<float*>(preds.mutable_data_ptr());
  void* s = stream_now();
  std::vector<hb_mlp_grid> grids;
  std::vector<hb_iteration_kind> its;
  for (const Kind& k : kinds) {
    const bool predict = k.blocks > 1;
    its.push_back(hb_iteration_kind{static_cast<const float*>(data(k.ms)), predict ? p : nullptr,
                                    static_cast<const int64_t*>(data(k.off)), k.f->size(0)});
    if (!predict) continue;
    grids.push_back(hb_mlp_grid{k.h, static_cast<const float*>(data(k.f)), k.f->size(0), k.rows,
                                static_cast<int32_t>(k.blocks), p});
    p += (k.blocks * k.f->size(0) + 63) & ~int64_t{63};
  }
  hb_status st = HB_OK;
  Py_BEGIN_ALLOW_THREADS
  for (size_t i = 0; i < grids.size() && st == HB_OK; i += 4)
    st = api.mlp_predict_grid(grids.data() + i, static_cast<int32_t>(grids.size() - i < 4 ? grids.size() - i : 4), s);
  if (st == HB_OK)
    st = api.iteration_totals(static_cast<const float*>(data(over)), static_cast<const float*>(tm.ptr()),
                              static_cast<const float*>(data(scaled)), K, static_cast<const int64_t*>(data(off)), I,
                              static_cast<int32_t>(D), same, its.data(), static_cast<int32_t>(its.size()),
                              static_cast<double*>(out.mutable_data_ptr()), s);
  Py_END_ALLOW_THREADS
  if (failed(st)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// setup(addresses by name, row_of, check, WaveResult, DeviceProperties)
PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5 || !PyDict_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "setup(addresses, row_of, check, WaveResult, DeviceProperties)");
    return nullptr;
  }
  auto load = [&](auto& fn, const char* name) {
    PyObject* v = PyDict_GetItemString(a[0], name);   // borrowed
    fn = v ? reinterpret_cast<std::remove_reference_t<decltype(fn)>>(PyLong_AsVoidPtr(v)) : nullptr;
    return fn != nullptr;
  };
  if (!load(api.wave_scale, "hb_wave_scale") || !load(api.wave_scale_metrics, "hb_wave_scale_metrics") ||
      !load(api.wave_scale_partials, "hb_wave_scale_partials") ||
      !load(api.wave_scale_host, "hb_wave_scale_host") || !load(api.partials_sum, "hb_partials_sum") ||
      !load(api.mlp_predict, "hb_mlp_predict") || !load(api.mlp_predict_host, "hb_mlp_predict_host") || !load(api.group_sum, "hb_group_sum") ||
      !load(api.plane_sum, "hb_plane_sum") || !load(api.segment_sum, "hb_segment_sum") ||
      !load(api.segment_sum_planes, "hb_segment_sum_planes") ||
      !load(api.mlp_predict_grid, "hb_mlp_predict_grid") || !load(api.mlp_poll_status, "hb_mlp_poll_status") ||
      !load(api.special_scale_grid, "hb_special_scale_grid") ||
      !load(api.iteration_totals, "hb_iteration_totals")) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "an entry point is missing");
    return nullptr;
  }
  Py_XSETREF(g_row_of, Py_NewRef(a[1]));
  Py_XSETREF(g_raise, Py_NewRef(a[2]));
  Py_XSETREF(g_wave_result, Py_NewRef(a[3]));
  Py_XSETREF(g_device_type, Py_NewRef(a[4]));
  Py_RETURN_NONE;
}

PyObject* set_generation(PyObject*, PyObject* v) {
  g_generation = PyLong_AsLong(v);
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(setup), FAST(wave_scale), FAST(wave_scale_host), FAST(submit_wave), FAST(host_block), FAST(release_host_blocks), FAST(mlp_predict), FAST(mlp_predict_one), FAST(flatten_trace), FAST(start_kinds), FAST(run_group), FAST(iteration_totals), FAST(partials_sum), FAST(group_sum),
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
      {&s_buffer, "buffer"}, {&s_K, "K"}, {&s_D, "D"}, {&s_per_plane, "per_plane"}, {&s_n_planes, "n_planes"},
      {&s__name, "_name"}, {&s__device, "_device"}, {&s__forward, "_forward"}, {&s__backward, "_backward"},
      {&s__arguments, "_arguments"}, {&s_args, "args"}, {&s_kwargs, "kwargs"}, {&s__kernels, "_kernels"},
      {&s__run_time_ms, "_run_time_ms"}, {&s__c, "_c"}, {&s__metrics_kernels, "_metrics_kernels"},
      {&s__cached_metrics, "_cached_metrics"}, {&s__metrics, "_metrics"}, {&s__num_blocks, "_num_blocks"},
      {&s__block_size, "_block_size"}, {&s__regs, "_registers_per_thread"},
      {&s__smem_static, "_static_shared_memory"}, {&s__smem_dynamic, "_dynamic_shared_memory"},
      {&s__run_time_ns, "_run_time_ns"}, {&s_name, "name"}};
  for (const auto& n : names)
    if (!(*n.s = PyUnicode_InternFromString(n.name))) return nullptr;
  if (PyType_Ready(&host_block_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
