// Native front of the operators: the part of a call that is the same every time (argument checks, output allocation, stream and
// workspace lookup, the C call) without the interpreter.
//
// What bounds it: a small packed linear runs 5-15 us on the GPU, while the same steps in Python and ctypes took 26 us per call on
// the host (attribute reads of six tensors, a device context manager, 16 converted arguments), so calls queued behind the host.
// Here a call costs about the launch itself.
//
// Each function either enqueues the whole call and returns its result, or returns None having enqueued nothing that matters: a
// wrong type, device or shape, a tensor subclass, a tensor that is not contiguous, a workspace that is missing or too small, or a
// status of the library other than HTR_OK.  The caller then takes the general path (htr_b200/ops.py), which raises the error,
// copies the operand or makes the workspace.  Entry points of the library arrive as addresses (bind), so that this module and the
// ctypes binding use one loaded library.  Every function runs with the interpreter lock held: the launches of one call are never
// interleaved with those of another thread on the same workspace.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <optional>
#include <vector>

#include "../../include/htr_b200.h"

namespace {

struct Entry {
  decltype(&htr_linear_workspace_bytes) linear_workspace_bytes;
  decltype(&htr_linear_gemm_workspace_bytes) linear_gemm_workspace_bytes;
  decltype(&htr_linear_ex) linear_ex;
  decltype(&htr_linear_gemm) linear_gemm;
  decltype(&htr_linear_padded) linear_padded;
  decltype(&htr_linear_fused) linear_fused;
  decltype(&htr_linear_gemm_padded) linear_gemm_padded;
  decltype(&htr_linear_route_rows) route_rows;
  decltype(&htr_linear_routed) linear_routed;
  decltype(&htr_linear_routed_gemm) linear_routed_gemm;
  decltype(&htr_route_plan_bytes) route_plan_bytes;
  decltype(&htr_route_plan) route_plan;
  decltype(&htr_moe_weighted_sum) moe_weighted_sum;
  decltype(&htr_dec_rope_cache) rope_cache;
  decltype(&htr_dec_attention) attention;
  decltype(&htr_dec_rope_attention) rope_attention;
  decltype(&htr_dec_add_rmsnorm) add_rmsnorm;
  decltype(&htr_dec_swiglu) swiglu;
} g_lib = {};

// ---- workspaces: buffers that ops.py owns (one per device, stream and kind); this table only remembers where they are
enum Kind { kGemv = 0, kGemm = 1 };
struct Workspace {
  int kind, device;
  void* stream;
  at::Tensor buf;
};
std::vector<Workspace>& workspaces() {
  static auto* table = new std::vector<Workspace>();     // never destroyed: the CUDA context may be gone by then
  return *table;
}
const at::Tensor* find_workspace(int kind, int device, void* stream) {
  for (const Workspace& w : workspaces())
    if (w.stream == stream && w.device == device && w.kind == kind) return &w.buf;
  return nullptr;
}

const at::Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return HTR_DTYPE_BF16;
    case at::kHalf: return HTR_DTYPE_F16;
    case at::kFloat: return HTR_DTYPE_F32;
    default: return -1;
  }
}

bool plain(const at::Tensor& t, const at::Device& dev, at::ScalarType type) {
  return t.scalar_type() == type && t.device() == dev && t.is_contiguous();
}

// the four wire tensors of one linear
struct Weight {
  const void *qw, *sc;
  const uint8_t *su, *sv;
  int mt, nt, K;
};
bool weight(PyObject* const* a, const at::Device& dev, Weight* w) {
  const at::Tensor *qw = tensor(a[0]), *sc = tensor(a[1]), *su = tensor(a[2]), *sv = tensor(a[3]);
  if (!qw || !sc || !su || !sv) return false;
  if (!plain(*qw, dev, at::kInt) || !plain(*sc, dev, at::kHalf) || !plain(*su, dev, at::kByte) || !plain(*sv, dev, at::kByte)) return false;
  if (qw->dim() != 3 || qw->size(2) % 8 || qw->size(0) > (1 << 24) || qw->size(1) > (1 << 24)) return false;
  w->mt = (int)qw->size(0);
  w->nt = (int)qw->size(1);
  w->K = (int)(qw->size(2) / 8);
  if (sc->numel() != (int64_t)w->mt * 16 || su->numel() != (int64_t)w->nt * 2 || sv->numel() != (int64_t)w->mt * 2) return false;
  w->qw = qw->const_data_ptr();
  w->sc = sc->const_data_ptr();
  w->su = static_cast<const uint8_t*>(su->const_data_ptr());
  w->sv = static_cast<const uint8_t*>(sv->const_data_ptr());
  return true;
}

// None, or a bias of `count` elements of the activation type
bool bias_of(PyObject* o, const at::Tensor& x, int64_t count, const void** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* b = tensor(o);
  if (!b || !plain(*b, x.device(), x.scalar_type()) || b->numel() != count) return false;
  *out = b->const_data_ptr();
  return true;
}

at::Tensor output(const at::Tensor& x, int64_t columns) {
  c10::DimVector shape(x.sizes().begin(), x.sizes().end());
  shape.back() = columns;
  return at::detail::empty_cuda(shape, x.scalar_type(), x.device(), std::nullopt);
}

// the device of the activations becomes the current one for the call (a CUDAGuard costs two runtime calls: only when it has to)
struct OnDevice {
  std::optional<c10::cuda::CUDAGuard> guard;
  explicit OnDevice(int device) {
    if (c10::cuda::current_device() != device) guard.emplace((c10::DeviceIndex)device);
  }
};

PyObject* none() { Py_RETURN_NONE; }

// an argument that is a C int; false for anything else (another type, a value beyond its range), with no Python error left behind
bool int_of(PyObject* o, int* out) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *out = (int)v;
  return *out == v;
}
bool float_of(PyObject* o, double* out) {
  *out = PyFloat_AsDouble(o);
  if (*out == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// linear(x, qweight, scales, su, sv, bias, flags, gemv_rows, gemm_rows): up to gemv_rows activation rows as one GEMV, up to
// gemm_rows on the tensor-core GEMM
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 9) return none();
  const at::Tensor* x = tensor(a[0]);
  Weight w;
  const void* bias;
  if (!x || !x->is_cuda() || x->dim() < 1 || !x->is_contiguous() || !weight(a + 1, x->device(), &w)) return none();
  const int dt = dtype_code(x->scalar_type());
  const int64_t cols = (int64_t)w.nt * 16, rows64 = cols ? x->numel() / cols : 0;
  int flags, gemv_rows, gemm_rows;
  if (!int_of(a[6], &flags) || !int_of(a[7], &gemv_rows) || !int_of(a[8], &gemm_rows)) return none();
  if (dt < 0 || x->size(-1) != cols || rows64 < 1 || !bias_of(a[5], *x, (int64_t)w.mt * 16, &bias)) return none();
  // (the rule of ops._gemv_rows)
  int64_t most = gemv_rows;
  if (gemv_rows <= 4 && rows64 <= gemv_rows && gemm_rows > 0) most = std::min<int64_t>(most, g_lib.route_rows(dt, w.mt, w.nt, (unsigned)flags));
  const bool gemv = rows64 <= most && rows64 <= HTR_GEMV_MAX_ROWS;
  if (!gemv && (rows64 <= most || rows64 > gemm_rows)) return none();
  const int rows = (int)rows64, dev = x->get_device();
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* ws = find_workspace(gemv ? kGemv : kGemm, dev, st);
  if (!ws) return none();
  at::Tensor y = output(*x, (int64_t)w.mt * 16);
  const char* xp = static_cast<const char*>(x->const_data_ptr());
  char* yp = static_cast<char*>(y.data_ptr());
  if (gemv) {
    if (g_lib.linear_ex(xp, dt, rows, w.qw, w.mt, w.nt, w.K, w.sc, w.su, w.sv, bias, yp, ws->data_ptr(), ws->numel(), st, (unsigned)flags) != HTR_OK)
      return none();
  } else {
    const int step = dt == HTR_DTYPE_F32 ? HTR_GEMM_MAX_ROWS_F32 : HTR_GEMM_MAX_ROWS;
    const int64_t esize = x->element_size();
    for (int r = 0; r < rows; r += step) {
      const int here = rows - r < step ? rows - r : step;
      if (g_lib.linear_gemm(xp + r * cols * esize, dt, here, w.qw, w.mt, w.nt, w.K, w.sc, w.su, w.sv, bias, yp + (int64_t)r * w.mt * 16 * esize,
                            ws->data_ptr(), ws->numel(), st) != HTR_OK)
        return none();
    }
  }
  return THPVariable_Wrap(std::move(y));
}

// linear_padded(x, qweight, scales, su, sv, bias, m_out, gemv_rows): up to gemv_rows rows in GEMV launches, more on the tensor-core GEMM
PyObject* py_linear_padded(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8) return none();
  const at::Tensor* x = tensor(a[0]);
  Weight w;
  const void* bias;
  if (!x || !x->is_cuda() || x->dim() < 1 || !x->is_contiguous() || !weight(a + 1, x->device(), &w)) return none();
  const int dt = dtype_code(x->scalar_type());
  const int64_t n_in = x->size(-1);
  int m_out, gemv_rows;
  if (!int_of(a[6], &m_out) || !int_of(a[7], &gemv_rows)) return none();
  if (dt < 0 || n_in < 1 || n_in > (int64_t)w.nt * 16 || m_out < 1 || m_out > (int64_t)w.mt * 16 || !bias_of(a[5], *x, m_out, &bias)) return none();
  const int64_t rows = x->numel() / n_in, esize = x->element_size();
  if (rows < 1) return none();
  const int dev = x->get_device();
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const bool gemm = rows > gemv_rows;
  const at::Tensor* ws = find_workspace(gemm ? kGemm : kGemv, dev, st);
  if (!ws) return none();
  at::Tensor y = output(*x, m_out);
  const char* xp = static_cast<const char*>(x->const_data_ptr());
  char* yp = static_cast<char*>(y.data_ptr());
  const int64_t step = gemm ? HTR_GEMM_MAX_ROWS_F32 : HTR_GEMV_MAX_ROWS;
  const auto launch = gemm ? g_lib.linear_gemm_padded : g_lib.linear_padded;
  for (int64_t r = 0; r < rows; r += step) {
    const int here = (int)(rows - r < step ? rows - r : step);
    if (launch(xp + r * n_in * esize, dt, here, (int)n_in, w.qw, w.mt, w.nt, w.K, w.sc, w.su, w.sv, bias, yp + r * m_out * esize,
               m_out, ws->data_ptr(), ws->numel(), st) != HTR_OK)
      return none();
  }
  return THPVariable_Wrap(std::move(y));
}

// linear_fused(x2, qweight, scales, su, sv, out, prologue, norm_weight, eps, residual)
PyObject* py_linear_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10) return none();
  const at::Tensor* x = tensor(a[0]);
  Weight w;
  if (!x || !x->is_cuda() || x->dim() != 2 || x->scalar_type() != at::kBFloat16 || !x->is_contiguous() || !weight(a + 1, x->device(), &w)) return none();
  int prologue;
  double eps;
  if (!int_of(a[6], &prologue) || !float_of(a[8], &eps)) return none();
  const int truth = PyObject_IsTrue(a[9]);
  if (truth < 0) { PyErr_Clear(); return none(); }
  const bool residual = truth == 1;
  const int64_t rows = x->size(0), cols = (int64_t)w.nt * 16 * (prologue == HTR_PROLOGUE_SWIGLU ? 2 : 1), m = (int64_t)w.mt * 16;
  if (rows < 1 || rows > HTR_GEMV_MAX_ROWS || x->size(1) != cols) return none();
  const void* norm = nullptr;
  if (a[7] != Py_None) {
    const at::Tensor* g = tensor(a[7]);
    if (!g || !plain(*g, x->device(), at::kBFloat16) || g->numel() != (int64_t)w.nt * 16) return none();
    norm = g->const_data_ptr();
  }
  const int dev = x->get_device();
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* ws = find_workspace(kGemv, dev, st);
  if (!ws) return none();
  at::Tensor y;
  if (a[5] == Py_None) {
    if (residual) return none();
    y = output(*x, m);
  } else {
    const at::Tensor* o = tensor(a[5]);
    if (!o || !plain(*o, x->device(), at::kBFloat16) || o->dim() != 2 || o->size(0) != rows || o->size(1) != m) return none();
    y = *o;
  }
  if (g_lib.linear_fused(x->const_data_ptr(), (int)rows, w.qw, w.mt, w.nt, w.K, w.sc, w.su, w.sv, y.data_ptr(), ws->data_ptr(), ws->numel(), st,
                         prologue, norm, (float)eps, residual ? 1 : 0) != HTR_OK)
    return none();
  if (a[5] != Py_None) return Py_NewRef(a[5]);
  return THPVariable_Wrap(std::move(y));
}

// ---- the launches of a mixture-of-experts step (two linears and a sum: in Python and ctypes 54 us of host work, more than the GPU
// needs for a few tokens of small experts)

bool vector_of(const at::Tensor* t, const at::Device& dev, at::ScalarType type) { return t && t->dim() == 1 && plain(*t, dev, type); }

// four address tables of one length
bool tables_of(PyObject* const* a, const at::Device& dev, const at::Tensor* (&t)[4]) {
  for (int i = 0; i < 4; ++i) {
    t[i] = tensor(a[i]);
    if (!vector_of(t[i], dev, at::kLong) || t[i]->numel() != t[0]->numel() || t[i]->numel() > (1 << 24)) return false;
  }
  return true;
}

// linear_routed(x, route, four tables, mt, nt, K, x_div, prologue, out or None)
PyObject* py_linear_routed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 12) return none();
  const at::Tensor *x = tensor(a[0]), *route = tensor(a[1]), *t[4];
  if (!x || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous()) return none();
  const at::Device where = x->device();
  if (!vector_of(route, where, at::kLong) || !tables_of(a + 2, where, t)) return none();
  const int dt = dtype_code(x->scalar_type());
  int mt, nt, K, x_div, prologue;
  if (!int_of(a[6], &mt) || !int_of(a[7], &nt) || !int_of(a[8], &K) || !int_of(a[9], &x_div) || !int_of(a[10], &prologue)) return none();
  const int64_t count = route->numel();
  if (dt < 0 || count < 1 || count > (1 << 24) || mt < 1 || mt > (1 << 24) || nt < 1 || nt > (1 << 24) || x_div < 1 || x_div > (1 << 24)) return none();
  const int dev = x->get_device();
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* ws = find_workspace(kGemv, dev, st);
  if (!ws) return none();
  at::Tensor y;
  if (a[11] == Py_None) {
    y = at::detail::empty_cuda({count, (int64_t)mt * 16}, x->scalar_type(), where, std::nullopt);
  } else {
    const at::Tensor* o = tensor(a[11]);
    if (!o || !plain(*o, where, x->scalar_type()) || o->dim() != 2 || o->size(0) != count || o->size(1) != mt * 16) return none();
    y = *o;
  }
  if (g_lib.linear_routed(x->const_data_ptr(), dt, x_div, x->size(1), route->const_data_ptr<int64_t>(), (int)count, (int)t[0]->numel(),
                          static_cast<const void* const*>(t[0]->const_data_ptr()), static_cast<const void* const*>(t[1]->const_data_ptr()),
                          static_cast<const uint8_t* const*>(t[2]->const_data_ptr()), static_cast<const uint8_t* const*>(t[3]->const_data_ptr()), mt,
                          nt, K, y.data_ptr(), prologue, ws->data_ptr(), ws->numel(), st) != HTR_OK)
    return none();
  if (a[11] != Py_None) return Py_NewRef(a[11]);
  return THPVariable_Wrap(std::move(y));
}

// linear_routed_gemm(x, plan, count, four tables, mt, nt, K, x_div, prologue)
PyObject* py_linear_routed_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 12) return none();
  const at::Tensor *x = tensor(a[0]), *plan = tensor(a[1]), *t[4];
  if (!x || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous()) return none();
  const at::Device where = x->device();
  if (!vector_of(plan, where, at::kByte) || !tables_of(a + 3, where, t)) return none();
  const int dt = dtype_code(x->scalar_type());
  int count, mt, nt, K, x_div, prologue;
  if (!int_of(a[2], &count) || !int_of(a[7], &mt) || !int_of(a[8], &nt) || !int_of(a[9], &K) || !int_of(a[10], &x_div) || !int_of(a[11], &prologue))
    return none();
  if (dt < 0 || count < 1 || count > (1 << 24) || mt < 1 || mt > (1 << 24) || nt < 1 || nt > (1 << 24) || x_div < 1 || x_div > (1 << 24)) return none();
  if ((size_t)plan->numel() < g_lib.route_plan_bytes(count, (int)t[0]->numel())) return none();
  const int dev = x->get_device();
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* ws = find_workspace(kGemm, dev, st);
  if (!ws) return none();
  at::Tensor y = at::detail::empty_cuda({(int64_t)count, (int64_t)mt * 16}, x->scalar_type(), where, std::nullopt);
  if (g_lib.linear_routed_gemm(x->const_data_ptr(), dt, x_div, x->size(1), plan->const_data_ptr(), count, (int)t[0]->numel(),
                               static_cast<const void* const*>(t[0]->const_data_ptr()), static_cast<const void* const*>(t[1]->const_data_ptr()),
                               static_cast<const uint8_t* const*>(t[2]->const_data_ptr()), static_cast<const uint8_t* const*>(t[3]->const_data_ptr()), mt,
                               nt, K, y.data_ptr(), prologue, ws->data_ptr(), ws->numel(), st) != HTR_OK)
    return none();
  return THPVariable_Wrap(std::move(y));
}

// route_plan(route, four tables)
PyObject* py_route_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) return none();
  const at::Tensor *route = tensor(a[0]), *t[4];
  if (!route || !route->is_cuda() || !vector_of(route, route->device(), at::kLong) || !tables_of(a + 1, route->device(), t)) return none();
  const int64_t count = route->numel(), rows = t[0]->numel();
  const size_t need = count < 1 || count > (1 << 24) ? 0 : g_lib.route_plan_bytes((int)count, (int)rows);
  if (need == 0) return none();
  const int dev = route->get_device();
  OnDevice on(dev);
  at::Tensor plan = at::detail::empty_cuda({(int64_t)need}, at::kByte, route->device(), std::nullopt);
  if (g_lib.route_plan(route->const_data_ptr<int64_t>(), (int)count, (int)rows, static_cast<const void* const*>(t[0]->const_data_ptr()), plan.data_ptr(),
                       need, c10::cuda::getCurrentCUDAStream(dev).stream()) != HTR_OK)
    return none();
  return THPVariable_Wrap(std::move(plan));
}

// moe_weighted_sum(dn [T * k, h], gates [T, k] float32)
PyObject* py_moe_weighted_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) return none();
  const at::Tensor *dn = tensor(a[0]), *gates = tensor(a[1]);
  if (!dn || !gates || !dn->is_cuda() || dn->dim() != 2 || !dn->is_contiguous() || !plain(*gates, dn->device(), at::kFloat) || gates->dim() != 2) return none();
  const int dt = dtype_code(dn->scalar_type());
  const int64_t T = gates->size(0), k = gates->size(1), h = dn->size(1);
  if (dt < 0 || T < 1 || T > (1 << 24) || k > (1 << 24) || h > (1 << 24) || dn->size(0) != T * k) return none();
  const int dev = dn->get_device();
  OnDevice on(dev);
  at::Tensor y = at::detail::empty_cuda({T, h}, dn->scalar_type(), dn->device(), std::nullopt);
  if (g_lib.moe_weighted_sum(dn->const_data_ptr(), dt, gates->const_data_ptr<float>(), (int)T, (int)k, (int)h, y.data_ptr(),
                             c10::cuda::getCurrentCUDAStream(dev).stream()) != HTR_OK)
    return none();
  return THPVariable_Wrap(std::move(y));
}

// ---- a step of the decoder (the loops of PackedDecoder.forward_folded and forward_fused): a decode-sized one is five or six launches a layer, 85 us
// of host work in Python, more than the GPU needs for layers of small models; 24 here (two layers of hidden 1024, a token: 210 -> 95 us).
// Whatever could refuse a launch of the step (shapes, alignment, workspace) is looked at before the first one, so that None means that
// nothing is enqueued and x is as it was; a launch that fails all the same (a CUDA error) raises.

bool wire_of(PyObject* o, const at::Device& dev, Weight* w) {   // the tuple of four wire tensors
  PyObject* item[4];
  if (!o || !PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 4) return false;
  for (int i = 0; i < 4; ++i) item[i] = PyTuple_GET_ITEM(o, i);
  return weight(item, dev, w);
}

// decoder_step(x, layers, head, ln_f, k_cache, v_cache, pos, cos, sin, status, q_heads, kv_heads, eps, gemm_rows): logits; x is overwritten.
// gemm_rows 0: the glue folded into the GEMVs (up to 8 rows); else separate glue kernels between tensor-core GEMMs, up to that many rows
PyObject* py_decoder_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 14) return none();
  static PyObject *const kQkv = PyUnicode_InternFromString("qkv"), *const kO = PyUnicode_InternFromString("o"),
                  *const kUp = PyUnicode_InternFromString("gate_up"), *const kDown = PyUnicode_InternFromString("down"),
                  *const kLn1 = PyUnicode_InternFromString("ln1"), *const kLn2 = PyUnicode_InternFromString("ln2");
  const at::Tensor *x = tensor(a[0]), *kc = tensor(a[4]), *vc = tensor(a[5]), *pos = tensor(a[6]), *cosv = tensor(a[7]), *sinv = tensor(a[8]), *status = tensor(a[9]);
  if (!x || !kc || !vc || !pos || !cosv || !sinv || !status || !PyList_CheckExact(a[1]) || !x->is_cuda() || x->dim() != 2) return none();
  const at::Device where = x->device();
  int hq, hkv, gemm_rows;
  double eps;
  if (!int_of(a[10], &hq) || !int_of(a[11], &hkv) || !float_of(a[12], &eps) || !int_of(a[13], &gemm_rows)) return none();
  const bool folded = gemm_rows == 0;
  constexpr int64_t D = 128;
  const int64_t T = x->size(0), hidden = x->size(1);
  const Py_ssize_t count = PyList_GET_SIZE(a[1]);
  if (!plain(*x, where, at::kBFloat16) || T < 1 || T > (folded ? HTR_GEMV_MAX_ROWS : gemm_rows) || hq < 1 || hkv < 1 || hq > 4096 || hkv > hq) return none();
  if (!plain(*kc, where, at::kBFloat16) || !plain(*vc, where, at::kBFloat16) || kc->dim() != 4 || kc->sizes() != vc->sizes() || kc->size(0) < count ||
      kc->size(2) != hkv || kc->size(3) != D)
    return none();
  const int64_t cap = kc->size(1), layer_bytes = cap * hkv * D * 2;
  if (!vector_of(pos, where, at::kLong) || pos->numel() != T || !plain(*cosv, where, at::kFloat) || !plain(*sinv, where, at::kFloat) ||
      cosv->numel() < cap * D / 2 || sinv->numel() < cap * D / 2 || !plain(*status, where, at::kInt) || status->numel() < 1)
    return none();

  struct Layer { Weight qkv, o, up, down; const void *ln1, *ln2; };
  std::vector<Layer> layers;
  layers.reserve((size_t)count);
  const auto norm_of = [&](PyObject* o, const void** out) {
    const at::Tensor* g = o ? tensor(o) : nullptr;
    if (!g || !plain(*g, where, at::kBFloat16) || g->numel() != hidden) return false;
    *out = g->const_data_ptr();
    return true;
  };
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* d = PyList_GET_ITEM(a[1], i);
    Layer l;
    if (!PyDict_CheckExact(d) || !wire_of(PyDict_GetItem(d, kQkv), where, &l.qkv) || !wire_of(PyDict_GetItem(d, kO), where, &l.o) ||
        !wire_of(PyDict_GetItem(d, kUp), where, &l.up) || !wire_of(PyDict_GetItem(d, kDown), where, &l.down) || !norm_of(PyDict_GetItem(d, kLn1), &l.ln1) ||
        !norm_of(PyDict_GetItem(d, kLn2), &l.ln2))
      return none();
    if (l.qkv.nt * 16 != hidden || l.qkv.mt * 16 != (hq + 2 * hkv) * D || l.o.nt * 16 != hq * D || l.o.mt * 16 != hidden || l.up.nt * 16 != hidden ||
        l.up.mt != 2 * l.down.nt || l.down.mt * 16 != hidden)
      return none();
    if (!layers.empty() && l.up.mt != layers[0].up.mt) return none();
    layers.push_back(l);
  }
  Weight head;
  const void* ln_f;
  if (!wire_of(a[2], where, &head) || head.nt * 16 != hidden || !norm_of(a[3], &ln_f)) return none();

  const int dev = x->get_device(), rows = (int)T;
  OnDevice on(dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* ws = find_workspace(folded ? kGemv : kGemm, dev, st);
  if (!ws) return none();
  const auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  Weight fits[5] = {};                                    // per role, the shape looked at last: layers are mostly alike
  const auto serves = [&](const Weight& w, int role) {
    if (!a16(w.qw) || !a16(w.sc)) return false;
    if (w.mt == fits[role].mt && w.nt == fits[role].nt && w.K == fits[role].K) return true;
    if (w.mt % 8 || w.nt % 8 || w.mt / 8 >= 16383 || (int64_t)(w.mt / 8) * (w.nt / 4) > 0x3FFFFFFF) return false;   // (limits of the launches)
    for (int r = 0; r < rows; r += folded ? rows : (int)HTR_GEMM_MAX_ROWS) {
      const size_t need = folded ? g_lib.linear_workspace_bytes(rows, w.mt * 16, w.nt * 16, w.K)
                                 : g_lib.linear_gemm_workspace_bytes(std::min(rows - r, (int)HTR_GEMM_MAX_ROWS), w.mt * 16, w.nt * 16, w.K);
      if (need == 0 || need > (size_t)ws->numel()) return false;
    }
    fits[role] = w;
    return true;
  };
  for (const Layer& l : layers)
    if (!serves(l.qkv, 0) || !serves(l.o, 1) || !serves(l.up, 2) || !serves(l.down, 3) || !a16(l.ln1) || !a16(l.ln2)) return none();
  if (!serves(head, 4) || !a16(ln_f) || !a16(x->const_data_ptr()) || hq % hkv || cap < 1 || (!folded && (hidden > 8192 || T > (1 << 16)))) return none();
  const auto failed = []() -> PyObject* { TORCH_CHECK(false, "decoder_step: a launch failed; part of the step is enqueued"); };
  const auto empty = [&](int64_t columns) { return at::detail::empty_cuda({T, columns}, at::kBFloat16, where, std::nullopt); };
  const at::Tensor qkv = empty((hq + 2 * hkv) * D), att = empty(hq * D), q = T > 1 || !folded ? empty(hq * D) : at::Tensor();
  const at::Tensor gu = empty(count ? (int64_t)layers[0].up.mt * 16 : 0);
  at::Tensor y = empty((int64_t)head.mt * 16);
  const auto fused = [&](const void* in, const Weight& w, void* out, int prologue, const void* norm, int residual) {
    return g_lib.linear_fused(in, rows, w.qw, w.mt, w.nt, w.K, w.sc, w.su, w.sv, out, ws->data_ptr(), ws->numel(), st, prologue, norm, (float)eps,
                              residual) == HTR_OK;
  };
  const int64_t* at_pos = pos->const_data_ptr<int64_t>();
  const float *cp = cosv->const_data_ptr<float>(), *sp = sinv->const_data_ptr<float>();
  int* sw = status->data_ptr<int>();
  void* xp = x->data_ptr();
  if (!folded) {
    const int inter = count ? layers[0].down.nt * 16 : 0;
    const at::Tensor h = empty(hidden), delta = empty(hidden), act = empty(inter);
    const auto gemm = [&](const at::Tensor& in, const Weight& w, const at::Tensor& out) {
      for (int r = 0; r < rows; r += HTR_GEMM_MAX_ROWS)
        if (g_lib.linear_gemm(static_cast<const char*>(in.const_data_ptr()) + (int64_t)r * w.nt * 32, HTR_DTYPE_BF16, std::min(rows - r, (int)HTR_GEMM_MAX_ROWS), w.qw,
                              w.mt, w.nt, w.K, w.sc, w.su, w.sv, nullptr, static_cast<char*>(out.data_ptr()) + (int64_t)r * w.mt * 32, ws->data_ptr(),
                              ws->numel(), st) != HTR_OK)
          return false;
      return true;
    };
    const auto norm = [&](const void* add, const void* gain) {
      return g_lib.add_rmsnorm(xp, add, gain, h.data_ptr(), rows, (int)hidden, (float)eps, st) == HTR_OK;
    };
    for (Py_ssize_t i = 0; i < count; ++i) {
      const Layer& l = layers[i];
      void *kl = static_cast<char*>(kc->data_ptr()) + i * layer_bytes, *vl = static_cast<char*>(vc->data_ptr()) + i * layer_bytes;
      if (!norm(i ? delta.data_ptr() : nullptr, l.ln1) || !gemm(h, l.qkv, qkv)) return failed();
      if (g_lib.rope_cache(qkv.data_ptr(), at_pos, cp, sp, q.data_ptr(), kl, vl, rows, hq, hkv, (int)D, (int)cap, sw, st) != HTR_OK) return failed();
      if (g_lib.attention(q.data_ptr(), kl, vl, at_pos, att.data_ptr(), rows, hq, hkv, (int)D, (int)cap, sw, st) != HTR_OK) return failed();
      if (!gemm(att, l.o, delta) || !norm(delta.data_ptr(), l.ln2) || !gemm(h, l.up, gu)) return failed();
      if (g_lib.swiglu(gu.data_ptr(), act.data_ptr(), rows, inter, st) != HTR_OK || !gemm(act, l.down, delta)) return failed();
    }
    if (!norm(count ? delta.data_ptr() : nullptr, ln_f) || !gemm(h, head, y)) return failed();
    return THPVariable_Wrap(std::move(y));
  }
  for (Py_ssize_t i = 0; i < count; ++i) {
    const Layer& l = layers[i];
    void *kl = static_cast<char*>(kc->data_ptr()) + i * layer_bytes, *vl = static_cast<char*>(vc->data_ptr()) + i * layer_bytes;
    if (!fused(xp, l.qkv, qkv.data_ptr(), HTR_PROLOGUE_RMSNORM, l.ln1, 0)) return failed();
    if (T == 1) {                                         // one token: rotary embedding, cache write and attention in one launch
      if (g_lib.rope_attention(qkv.data_ptr(), at_pos, cp, sp, kl, vl, att.data_ptr(), hq, hkv, (int)D, (int)cap, sw, st) != HTR_OK) return failed();
    } else {
      if (g_lib.rope_cache(qkv.data_ptr(), at_pos, cp, sp, q.data_ptr(), kl, vl, rows, hq, hkv, (int)D, (int)cap, sw, st) != HTR_OK) return failed();
      if (g_lib.attention(q.data_ptr(), kl, vl, at_pos, att.data_ptr(), rows, hq, hkv, (int)D, (int)cap, sw, st) != HTR_OK) return failed();
    }
    if (!fused(att.data_ptr(), l.o, xp, HTR_PROLOGUE_NONE, nullptr, 1) || !fused(xp, l.up, gu.data_ptr(), HTR_PROLOGUE_RMSNORM, l.ln2, 0) ||
        !fused(gu.data_ptr(), l.down, xp, HTR_PROLOGUE_SWIGLU, nullptr, 1))
      return failed();
  }
  if (!fused(xp, head, y.data_ptr(), HTR_PROLOGUE_RMSNORM, ln_f, 0)) return failed();
  return THPVariable_Wrap(std::move(y));
}

// set_workspace(kind, device index, stream, buffer): the buffer that calls on this device and stream use from now on
PyObject* py_set_workspace(PyObject*, PyObject* args) {
  int kind, device;
  unsigned long long stream;
  PyObject* buf;
  if (!PyArg_ParseTuple(args, "iiKO", &kind, &device, &stream, &buf)) return nullptr;
  if (!THPVariable_Check(buf)) {
    PyErr_SetString(PyExc_TypeError, "set_workspace wants a tensor");
    return nullptr;
  }
  void* st = reinterpret_cast<void*>(stream);
  for (Workspace& w : workspaces())
    if (w.stream == st && w.device == device && w.kind == kind) {
      w.buf = THPVariable_Unpack(buf);
      Py_RETURN_NONE;
    }
  workspaces().push_back({kind, device, st, THPVariable_Unpack(buf)});
  Py_RETURN_NONE;
}

// bind(dict name -> address of the loaded library's entry point)
PyObject* py_bind(PyObject*, PyObject* table) {
  const auto at_name = [&](const char* name) -> void* {
    PyObject* v = PyDict_Check(table) ? PyDict_GetItemString(table, name) : nullptr;
    return v ? PyLong_AsVoidPtr(v) : nullptr;
  };
  g_lib.linear_workspace_bytes = reinterpret_cast<decltype(g_lib.linear_workspace_bytes)>(at_name("htr_linear_workspace_bytes"));
  g_lib.linear_gemm_workspace_bytes = reinterpret_cast<decltype(g_lib.linear_gemm_workspace_bytes)>(at_name("htr_linear_gemm_workspace_bytes"));
  g_lib.linear_ex = reinterpret_cast<decltype(g_lib.linear_ex)>(at_name("htr_linear_ex"));
  g_lib.linear_gemm = reinterpret_cast<decltype(g_lib.linear_gemm)>(at_name("htr_linear_gemm"));
  g_lib.linear_padded = reinterpret_cast<decltype(g_lib.linear_padded)>(at_name("htr_linear_padded"));
  g_lib.linear_fused = reinterpret_cast<decltype(g_lib.linear_fused)>(at_name("htr_linear_fused"));
  g_lib.linear_gemm_padded = reinterpret_cast<decltype(g_lib.linear_gemm_padded)>(at_name("htr_linear_gemm_padded"));
  g_lib.route_rows = reinterpret_cast<decltype(g_lib.route_rows)>(at_name("htr_linear_route_rows"));
  g_lib.linear_routed = reinterpret_cast<decltype(g_lib.linear_routed)>(at_name("htr_linear_routed"));
  g_lib.linear_routed_gemm = reinterpret_cast<decltype(g_lib.linear_routed_gemm)>(at_name("htr_linear_routed_gemm"));
  g_lib.route_plan_bytes = reinterpret_cast<decltype(g_lib.route_plan_bytes)>(at_name("htr_route_plan_bytes"));
  g_lib.route_plan = reinterpret_cast<decltype(g_lib.route_plan)>(at_name("htr_route_plan"));
  g_lib.moe_weighted_sum = reinterpret_cast<decltype(g_lib.moe_weighted_sum)>(at_name("htr_moe_weighted_sum"));
  g_lib.rope_cache = reinterpret_cast<decltype(g_lib.rope_cache)>(at_name("htr_dec_rope_cache"));
  g_lib.attention = reinterpret_cast<decltype(g_lib.attention)>(at_name("htr_dec_attention"));
  g_lib.rope_attention = reinterpret_cast<decltype(g_lib.rope_attention)>(at_name("htr_dec_rope_attention"));
  g_lib.add_rmsnorm = reinterpret_cast<decltype(g_lib.add_rmsnorm)>(at_name("htr_dec_add_rmsnorm"));
  g_lib.swiglu = reinterpret_cast<decltype(g_lib.swiglu)>(at_name("htr_dec_swiglu"));
  if (!g_lib.linear_workspace_bytes || !g_lib.linear_gemm_workspace_bytes || !g_lib.add_rmsnorm || !g_lib.swiglu || !g_lib.rope_cache || !g_lib.attention || !g_lib.rope_attention || !g_lib.linear_routed || !g_lib.linear_routed_gemm || !g_lib.route_plan_bytes || !g_lib.route_plan || !g_lib.moe_weighted_sum ||
      !g_lib.linear_gemm_padded || !g_lib.route_rows || !g_lib.linear_ex || !g_lib.linear_gemm || !g_lib.linear_padded || !g_lib.linear_fused) {
    PyErr_SetString(PyExc_ImportError, "bind: an entry point of libhtr_b200 is missing");
    return nullptr;
  }
  Py_RETURN_NONE;
}

// C++ exceptions (out of memory in the allocator, a sticky CUDA error) become the Python exceptions torch uses
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef fast(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<F>)), METH_FASTCALL, nullptr};
}

PyMethodDef g_methods[] = {
    fast<py_linear>("linear"),
    fast<py_linear_padded>("linear_padded"),
    fast<py_linear_fused>("linear_fused"),
    fast<py_linear_routed>("linear_routed"),
    fast<py_linear_routed_gemm>("linear_routed_gemm"),
    fast<py_route_plan>("route_plan"),
    fast<py_moe_weighted_sum>("moe_weighted_sum"),
    fast<py_decoder_step>("decoder_step"),
    {"set_workspace", py_set_workspace, METH_VARARGS, nullptr},
    {"bind", py_bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host", "native front of the packed-linear operators", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&g_module); }
