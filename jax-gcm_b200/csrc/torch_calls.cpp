// torch_calls.cpp -- the plain calls on torch tensors: gathers the field pointers, allocates the
// results and calls the C ABI, for physics.py, adjoint.py, held_suarez.py and rollout.py.
//
// A small call is bound by the host: through ctypes (ctypes_calls.py, the same calls for a torch that
// this module has not been built for) a T21 call with its diagnostics took 91 us, of which the
// device works 17 (21 torch.empty calls of 2.4 us each, 38 pointers, the structures).  Through this
// module it takes 37 us (T85 with 16 levels 45 -> 24, a 361 x 181 Held-Suarez call 27 -> 16; a T42
// VJP with 8 levels 44 -> 28.7, which the device bounds); 21 of the 37 are the 21 result tensors.
// It does the same in one call: 17 attribute reads and checks, one allocation per result through
// torch's allocator, and the library call with the interpreter's lock released.  Nothing is kept
// between calls.  The library's entry points come in as addresses (bind), so that this module does
// not depend on which build of the library is loaded.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include <array>

#include "speedy_b200.h"

namespace {

decltype(&spd_fwd_marked) g_fwd = nullptr;
decltype(&spd_vjp) g_vjp = nullptr;
decltype(&spd_held_suarez) g_hs = nullptr;
decltype(&spd_rollout_step) g_step = nullptr;
decltype(&spd_rollout_reverse) g_reverse = nullptr;

enum Owner { kState, kForcing, kGeometry };
struct Name {
  const char* text;
  Owner owner;
  PyObject* str;
};
// spd_inputs_t in order.
Name g_inputs[] = {{"u_wind", kState, nullptr}, {"v_wind", kState, nullptr},
                   {"temperature", kState, nullptr}, {"specific_humidity", kState, nullptr},
                   {"geopotential", kState, nullptr},
                   {"normalized_surface_pressure", kState, nullptr}, {"alb0", kForcing, nullptr},
                   {"sice_am", kForcing, nullptr}, {"snowc_am", kForcing, nullptr},
                   {"soilw_am", kForcing, nullptr}, {"stl_am", kForcing, nullptr},
                   {"sea_surface_temperature", kForcing, nullptr}, {"fmask", kGeometry, nullptr},
                   {"orog", kGeometry, nullptr}, {"phis0", kGeometry, nullptr},
                   {"sia", kGeometry, nullptr}, {"coa", kGeometry, nullptr}};
constexpr int kInputs = sizeof(g_inputs) / sizeof(g_inputs[0]);
static_assert(kInputs * sizeof(void*) == sizeof(spd_inputs_t), "one pointer per input field");
constexpr int kOutputs = sizeof(spd_outputs_t) / sizeof(void*);
constexpr int kLevelInputs = 5, kLatitudeInputs = 2;  // the first ones, and the last
const char* const g_outputs[] = {"u_wind", "v_wind", "temperature", "specific_humidity", "precnv",
                                 "precls", "cbmf", "cloudc", "cloudstr", "rsds", "rsns", "ftop_sw",
                                 "rlds", "rlns", "ftop_lw", "tsfc", "tskin", "shf", "evap",
                                 "iptop", "icltop"};
static_assert(sizeof(g_outputs) / sizeof(g_outputs[0]) == kOutputs, "one name per output field");
constexpr int kLevelOutputs = 4, kFloatOutputs = 19, kPlainOutputs = 6;

// The kernels' extents come from the geometry, not from the tensors: a field has to hold the values
// that they read, and a result the bytes that they write.
void expect_values(const at::Tensor& t, int64_t need, const char* name) {
  TORCH_CHECK_VALUE(t.numel() >= need, name, " has ", t.numel(), " values, the geometry has ", need);
}
void expect_room(const at::Tensor& t, int64_t need, const char* name) {
  const int64_t room =
      (int64_t)t.storage().nbytes() - t.storage_offset() * (int64_t)t.element_size();
  TORCH_CHECK_VALUE(room >= need * 4, name, " (out) has room for ", room / 4,
                    " values, the geometry has ", need);
}
void expect_device(const at::Tensor& t) {
  TORCH_CHECK(t.is_cuda() || t.is_pinned(), "out holds CUDA tensors");
}

at::Tensor attribute(PyObject* obj, PyObject* name) {
  PyObject* v = PyObject_GetAttr(obj, name);
  if (!v) throw python_error();
  const bool is = THPVariable_Check(v);
  at::Tensor t = is ? THPVariable_Unpack(v) : at::Tensor();
  Py_DECREF(v);
  TORCH_CHECK_TYPE(is, PyUnicode_AsUTF8(name), " must be a tensor");
  return t;
}

// `t` as contiguous float32 on `device`; itself where it is that already.
at::Tensor as_input(at::Tensor t, c10::Device device) {
  if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.device() != device)
    return t.to(device, at::kFloat).contiguous();
  return t;
}

c10::Device device_of(PyObject* state, int temperature = 2) {
  return attribute(state, g_inputs[temperature].str).device();
}

struct Fields {
  std::array<at::Tensor, kInputs> t;  // keeps converted copies until the call is enqueued
  spd_inputs_t in;
};

// low_winds: u and v are planes of the lowest level.
Fields fields(PyObject* state, PyObject* forcing, PyObject* geometry, c10::Device device,
              const spd_desc_t* desc, bool low_winds) {
  const int64_t columns = (int64_t)desc->ix * desc->il, level = desc->kx * columns;
  PyObject* const owners[] = {state, forcing, geometry};
  Fields f;
  const float** p = reinterpret_cast<const float**>(&f.in);
  for (int i = 0; i < kInputs; ++i) {
    at::Tensor t = attribute(owners[g_inputs[i].owner], g_inputs[i].str);
    expect_values(t, i >= kInputs - kLatitudeInputs                       ? desc->il
                     : i < kLevelInputs && !(low_winds && i < 2) ? level
                                                                 : columns,
                  g_inputs[i].text);
    f.t[i] = as_input(std::move(t), device);
    p[i] = static_cast<const float*>(f.t[i].const_data_ptr());
  }
  return f;
}

// A result tensor, from torch's caching allocator.
at::Tensor empty(at::IntArrayRef shape, c10::Device device, at::ScalarType type = at::kFloat) {
  return at::detail::empty_cuda(shape, type, device, std::nullopt);
}

template <class T>
T* address(PyObject* v) {
  void* p = PyLong_AsVoidPtr(v);
  if (!p && PyErr_Occurred()) throw python_error();
  return static_cast<T*>(p);
}

void* stream_of(c10::Device device) {
  return c10::cuda::getCurrentCUDAStream(device.index()).stream();
}

PyObject* result(int rc, const at::Tensor* t, int n) {
  PyObject* list = PyList_New(n);
  if (!list) throw python_error();
  for (int i = 0; i < n; ++i) {
    PyObject* v = t[i].defined() ? THPVariable_Wrap(t[i]) : (Py_INCREF(Py_None), Py_None);
    PyList_SET_ITEM(list, i, v);
  }
  return Py_BuildValue("(iN)", rc, list);
}

void expect(Py_ssize_t have, Py_ssize_t want) {
  TORCH_CHECK_TYPE(have == want, "expected ", want, " arguments, got ", have);
}

// fwd(state, forcing, geometry, out, diagnostics, desc, vgrid, params, scratch, scratch_bytes,
//     event) -> (status, [tensor or None per spd_outputs_t field])
// out: None, or a list of tensors or None in spd_outputs_t's order.
PyObject* fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 11);
  const auto* desc = address<const spd_desc_t>(a[5]);
  const c10::Device device = device_of(a[0]);
  const bool low_winds = (desc->flags & SPD_LOW_LEVEL_WINDS) != 0;
  Fields f = fields(a[0], a[1], a[2], device, desc, low_winds);
  const int64_t columns = (int64_t)desc->ix * desc->il;
  std::array<at::Tensor, kOutputs> t;
  spd_outputs_t out{};
  void** p = reinterpret_cast<void**>(&out);
  if (a[3] != Py_None) {
    TORCH_CHECK_TYPE(PyList_Check(a[3]) && PyList_GET_SIZE(a[3]) == kOutputs, "out is a list");
    for (int i = 0; i < kOutputs; ++i) {
      PyObject* v = PyList_GET_ITEM(a[3], i);
      if (v == Py_None) continue;
      TORCH_CHECK_TYPE(THPVariable_Check(v), "out holds tensors");
      t[i] = THPVariable_Unpack(v);
      expect_room(t[i], i < kLevelOutputs && !(low_winds && i < 2) ? desc->kx * columns : columns,
                  g_outputs[i]);
    }
  }
  TORCH_CHECK(device.is_cuda(), "the physics runs on CUDA tensors only (no CPU path)");
  if (a[3] == Py_None) {
    const int64_t level[] = {desc->kx, desc->ix, desc->il}, surface[] = {desc->ix, desc->il};
    const int count = PyObject_IsTrue(a[4]) == 1 ? kOutputs : kPlainOutputs;
    for (int i = 0; i < count; ++i)
      t[i] = i < kLevelOutputs ? empty(level, device)
                               : empty(surface, device, i < kFloatOutputs ? at::kFloat : at::kInt);
  }
  for (int i = 0; i < kOutputs; ++i) {
    if (!t[i].defined()) continue;
    expect_device(t[i]);
    p[i] = t[i].data_ptr();
  }
  void* stream = stream_of(device);
  const auto* vgrid = address<const spd_vgrid_t>(a[6]);
  const auto* params = address<const spd_params_t>(a[7]);
  void* scratch = address<void>(a[8]);
  const size_t bytes = PyLong_AsSize_t(a[9]);
  void* event = address<void>(a[10]);
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = g_fwd(desc, vgrid, params, &f.in, &out, scratch, bytes, stream, event);
  }
  return result(rc, t.data(), kOutputs);
  END_HANDLE_TH_ERRORS
}

// vjp(state, forcing, geometry, cotangent, desc, vgrid, params, scratch_bytes)
//   -> (status, [u, v, T, q, phi, psa, params gradients])
// The scratch is the call's own, from torch's allocator on the current stream: calls on several
// streams or from several threads do not meet in it.
PyObject* vjp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 8);
  const auto* desc = address<const spd_desc_t>(a[4]);
  const c10::Device device = device_of(a[0]);
  Fields f = fields(a[0], a[1], a[2], device, desc, false);
  std::array<at::Tensor, 4> ct;
  spd_cotangents_t cot;
  const float** pc = reinterpret_cast<const float**>(&cot);
  for (int i = 0; i < 4; ++i) {
    at::Tensor t = attribute(a[3], g_inputs[i].str);
    expect_values(t, (int64_t)desc->kx * desc->ix * desc->il, g_inputs[i].text);
    ct[i] = as_input(std::move(t), device);
    pc[i] = static_cast<const float*>(ct[i].const_data_ptr());
  }
  TORCH_CHECK(device.is_cuda(), "the adjoint runs on CUDA tensors only (no CPU path)");
  std::array<at::Tensor, 7> g;
  spd_grads_t grads;
  float** pg = reinterpret_cast<float**>(&grads);
  for (int i = 0; i < 7; ++i) {
    g[i] = i < 6 ? empty(f.t[i].sizes(), device) : empty({SPD_NUM_DIFF_PARAMS}, device);
    pg[i] = static_cast<float*>(g[i].data_ptr());
  }
  void* stream = stream_of(device);
  const auto* vgrid = address<const spd_vgrid_t>(a[5]);
  const auto* params = address<const spd_params_t>(a[6]);
  const size_t bytes = PyLong_AsSize_t(a[7]);
  if (PyErr_Occurred()) throw python_error();
  const at::Tensor own = empty({(int64_t)bytes}, device, at::kByte);
  void* scratch = own.data_ptr();
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = g_vjp(desc, vgrid, params, &f.in, &cot, &grads, scratch, bytes, stream);
  }
  return result(rc, g.data(), 7);
  END_HANDLE_TH_ERRORS
}

// held_suarez(state, table, out, desc) -> (status, [du, dv, dT, dq]); out: None or four tensors.
PyObject* held_suarez(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  const c10::Device device = device_of(a[0]);
  const auto* desc = address<const spd_hs_desc_t>(a[3]);
  const int64_t columns = (int64_t)desc->ix * desc->il, level = desc->kx * columns;
  const int which[] = {0, 1, 2, 5};  // u, v, T, psa
  std::array<at::Tensor, 4> in, out;
  for (int i = 0; i < 4; ++i) {
    at::Tensor t = attribute(a[0], g_inputs[which[i]].str);
    expect_values(t, i < 3 ? level : columns, g_inputs[which[i]].text);
    in[i] = as_input(std::move(t), device);
  }
  TORCH_CHECK_TYPE(THPVariable_Check(a[1]), "the latitude table is a tensor");
  const at::Tensor& table = THPVariable_Unpack(a[1]);
  TORCH_CHECK_VALUE(table.numel() == 3 * (int64_t)desc->il && table.is_contiguous() &&
                        table.scalar_type() == at::kFloat && table.device() == device,
                    "the latitude table has three values for each of the geometry's latitudes");
  for (int i = 0; i < 4 && a[2] != Py_None; ++i) {
    TORCH_CHECK_TYPE(PyList_Check(a[2]) && PyList_GET_SIZE(a[2]) == 4, "out is a list of four");
    PyObject* v = PyList_GET_ITEM(a[2], i);
    TORCH_CHECK_TYPE(THPVariable_Check(v), "out holds tensors");
    out[i] = THPVariable_Unpack(v);
    expect_room(out[i], level, g_outputs[i]);
  }
  TORCH_CHECK(device.is_cuda(), "HeldSuarezPhysics runs on CUDA tensors only (no CPU path)");
  for (at::Tensor& t : out) {
    if (!t.defined()) t = empty(in[2].sizes(), device);
    expect_device(t);
  }
  void* stream = stream_of(device);
  auto p = [](const at::Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); };
  auto w = [](const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); };
  const float* lat = p(table);
  const float *u = p(in[0]), *v = p(in[1]), *t = p(in[2]), *psa = p(in[3]);
  float *du = w(out[0]), *dv = w(out[1]), *dt = w(out[2]), *dq = w(out[3]);
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = g_hs(desc, lat, u, v, t, psa, du, dv, dt, dq, stream);
  }
  return result(rc, out.data(), 4);
  END_HANDLE_TH_ERRORS
}

// A tensor that is no more than its values in memory: not a subclass of torch.Tensor, with no
// forward-mode tangent, and with no dispatch key that an operation would have to see (a functorch
// wrapper, a pending negation).
bool plain(PyObject* v) {
  if (!THPVariable_CheckExact(v)) return false;
  const at::Tensor& t = THPVariable_Unpack(v);
  constexpr c10::DispatchKeySet seen({
      c10::DispatchKey::Negative, c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor,
      c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::Batched,
      c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
  return !t.key_set().has_any(seen) && !t._fw_grad(0).defined();
}

// The tensor attributes u_wind, v_wind, temperature and specific_humidity of an object (or the items
// of a list) when they are what the rollout's kernels take: plain contiguous float32 on one CUDA
// device, of one shape, with no gradient to record; false otherwise, and wherever a dispatch mode
// watches the operations.
bool planes(PyObject* obj, std::array<at::Tensor, 4>& t) {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  if (PyList_Check(obj) && PyList_GET_SIZE(obj) != 4) return false;
  for (int i = 0; i < 4; ++i) {
    const auto v = pybind11::reinterpret_steal<pybind11::object>(
        PyList_Check(obj) ? Py_NewRef(PyList_GET_ITEM(obj, i))
                          : PyObject_GetAttr(obj, g_inputs[i].str));
    if (!v) throw python_error();
    if (!plain(v.ptr())) return false;
    t[i] = THPVariable_Unpack(v.ptr());
    if (!t[i].is_cuda() || t[i].scalar_type() != at::kFloat || !t[i].is_contiguous() ||
        t[i].dim() < 1 || t[i].numel() == 0 || t[i].device() != t[0].device() ||
        t[i].sizes() != t[0].sizes() || (t[i].requires_grad() && c10::GradMode::is_enabled()))
      return false;
  }
  return true;
}

template <class S>
S pointers(const std::array<at::Tensor, 4>& t) {
  S s;
  auto** p = reinterpret_cast<void**>(&s);
  for (int i = 0; i < 4; ++i) p[i] = t[i].data_ptr();
  return s;
}

std::array<at::Tensor, 4> empty_planes(const at::Tensor& like) {
  std::array<at::Tensor, 4> t;
  for (at::Tensor& x : t) x = empty(like.sizes(), like.device());
  return t;
}

// rollout_step(state, tendency, dt) -> (status, [u, v, T, q]), or None where the planes are not
// what the kernel takes.
PyObject* rollout_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 3);
  std::array<at::Tensor, 4> x, f;
  if (!planes(a[0], x) || !planes(a[1], f) || x[0].sizes() != f[0].sizes() ||
      x[0].device() != f[0].device() || x[0].size(0) > SPD_MAX_KX)
    Py_RETURN_NONE;
  const double dt = PyFloat_AsDouble(a[2]);
  if (PyErr_Occurred()) throw python_error();
  const std::array<at::Tensor, 4> out = empty_planes(x[0]);
  const auto px = pointers<spd_cotangents_t>(x), pf = pointers<spd_cotangents_t>(f);
  const auto po = pointers<spd_planes_t>(out);
  const int32_t kx = (int32_t)x[0].size(0);
  const int64_t columns = x[0].numel() / kx;
  void* stream = stream_of(x[0].device());
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = g_step(kx, columns, (float)dt, &px, &pf, &po, stream);
  }
  return result(rc, out.data(), 4);
  END_HANDLE_TH_ERRORS
}

// rollout_reverse(xbar, gradients, params, phi_sum, psa_sum, params_sum, dt)
//   -> (status, [four xbar planes, four cotangent planes]), or None where they are not what the
// kernel takes.  xbar: four planes; gradients: a PhysicsState; the sums are added to in place.
PyObject* rollout_reverse(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 7);
  std::array<at::Tensor, 4> xb, g;
  if (!planes(a[0], xb) || !planes(a[1], g) || xb[0].sizes() != g[0].sizes() ||
      xb[0].device() != g[0].device() || xb[0].size(0) > SPD_MAX_KX)
    Py_RETURN_NONE;
  const at::Tensor g_phi = attribute(a[1], g_inputs[4].str), g_psa = attribute(a[1], g_inputs[5].str);
  std::array<at::Tensor, 6> rest = {g_phi, g_psa};
  for (int i = 0; i < 4; ++i) {
    TORCH_CHECK_TYPE(THPVariable_Check(a[2 + i]), "expected a tensor");
    rest[2 + i] = THPVariable_Unpack(a[2 + i]);
  }
  const int32_t kx = (int32_t)xb[0].size(0);
  const int64_t columns = xb[0].numel() / kx;
  const int64_t want[] = {kx * columns, columns, SPD_NUM_DIFF_PARAMS, kx * columns, columns,
                          SPD_NUM_DIFF_PARAMS};
  for (int i = 0; i < 6; ++i)
    if (rest[i].device() != xb[0].device() || rest[i].scalar_type() != at::kFloat ||
        !rest[i].is_contiguous() || rest[i].numel() != want[i])
      Py_RETURN_NONE;
  const double dt = PyFloat_AsDouble(a[6]);
  if (PyErr_Occurred()) throw python_error();
  std::array<at::Tensor, 8> t;
  const std::array<at::Tensor, 4> out = empty_planes(xb[0]), ct = empty_planes(xb[0]);
  for (int i = 0; i < 4; ++i) {
    t[i] = out[i];
    t[4 + i] = ct[i];
  }
  const auto px = pointers<spd_cotangents_t>(xb);
  const auto po = pointers<spd_planes_t>(out), pc = pointers<spd_planes_t>(ct);
  auto w = [&](int i) { return static_cast<float*>(rest[i].data_ptr()); };
  const spd_grads_t pg = {static_cast<float*>(g[0].data_ptr()), static_cast<float*>(g[1].data_ptr()),
                          static_cast<float*>(g[2].data_ptr()), static_cast<float*>(g[3].data_ptr()),
                          w(0), w(1), w(2)};
  float *phi = w(3), *psa = w(4), *par = w(5);
  void* stream = stream_of(xb[0].device());
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = g_reverse(kx, columns, (float)dt, &px, &pg, &po, &pc, phi, psa, par, stream);
  }
  return result(rc, t.data(), 8);
  END_HANDLE_TH_ERRORS
}

// bind(spd_fwd_marked, spd_vjp, spd_held_suarez, spd_rollout_step, spd_rollout_reverse): the
// library's entry points, as addresses.
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 5);
  g_fwd = reinterpret_cast<decltype(g_fwd)>(address<void>(a[0]));
  g_vjp = reinterpret_cast<decltype(g_vjp)>(address<void>(a[1]));
  g_hs = reinterpret_cast<decltype(g_hs)>(address<void>(a[2]));
  g_step = reinterpret_cast<decltype(g_step)>(address<void>(a[3]));
  g_reverse = reinterpret_cast<decltype(g_reverse)>(address<void>(a[4]));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef method(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL,
          nullptr};
}

PyMethodDef g_methods[] = {method<fwd>("fwd"), method<vjp>("vjp"),
                           method<held_suarez>("held_suarez"),
                           method<rollout_step>("rollout_step"),
                           method<rollout_reverse>("rollout_reverse"), method<bind>("bind"),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  for (Name& n : g_inputs)
    if (!(n.str = PyUnicode_InternFromString(n.text))) return nullptr;
  return PyModule_Create(&g_module);
}
